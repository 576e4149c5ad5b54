// True float32 matrix product: C[M,N] = A[M,K] * W[N,K]^T.
//
// This is the matrix product of the 32-bit path; no reduced-precision mode.  From K = 512 on the products run
// on the tensor cores without giving up a bit of an operand: every float32 number (times 2^16, see take_apart) is the
// exact sum of three bfloat16 numbers (8 bits each; rounded to nearest, what is left, what is left of that), and of the nine
// products of two such sums the six that matter are formed, the smallest first; the three left out are below
// 2^-25 of the product.  k is cut into blocks of 64 and these into four runs.  The tensor core sums a
// block from zero, in float32; a run adds its blocks up in index order with float32 additions outside the tensor
// core, and the runs are added in order.  Below K = 512 an element is one chain of FMA over k in index order
// (gemm_fp32_short_kernel).  The order is a function of K alone, whatever the tile, so a row's result does not
// depend on M: the same token gives the same bits in any batch.  A result that comes out as no finite number is formed
// again by FMA from the operands: an infinity is no sum of three numbers, and neither are operands above 2^112 or sums above
// 2^96, which the factor takes beyond float32's range.
// (Distance from 64-bit sums at K = 1,024 .. 4,096: 0.97e-7 .. 1.1e-7 of the norm, where eight chains of FMA had 2.1e-7 ..
// 4.1e-7.)
#include "common.cuh"

namespace {

constexpr int WARPS = 8;
constexpr int THREADS = WARPS * 32;

// rows r0 .. r0 + ROWS - 1 (below `rows`), k0 .. k0 + COLS - 1 (below K) of a [rows, K] matrix; zeros elsewhere
template <int ROWS, int COLS, int LD, bool VEC>
__device__ __forceinline__ void copy_rows(float* dst, const float* __restrict__ src, int r0, int rows, int k0, int K) {
  constexpr int E = VEC ? 4 : 1, PER = COLS / E;            // elements a copy, copies a row
  for (int i = threadIdx.x; i < ROWS * PER; i += THREADS) {
    const int r = i / PER, k = (i % PER) * E;
    const bool in = r0 + r < rows && k0 + k < K;
    const float* s = in ? src + (size_t)(r0 + r) * K + k0 + k : src;
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst + r * LD + k);
    if (VEC)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(s), "r"(in ? 16 : 0) : "memory");
    else
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(s), "r"(in ? 4 : 0) : "memory");
  }
}

// ---- tensor-core form.  A CTA takes 128 rows of W (the instruction's rows) by TOK rows of A (its columns) over a
// run of k or all of them (Form).  Per block of 64 k: every thread takes apart the numbers it asked for one or two blocks
// earlier and leaves the three parts of both operands in shared memory in the layout the instruction reads (rows of 128
// bytes, 128-byte swizzle), one more thread issues the 24 products into one of two accumulators in tensor memory (a warp of
// its own: it waits while the unit is busy), and while they run the accumulator of the block before is added to the sums in
// registers.  At the end the cluster's CTAs add their sums through one another's shared memory, in run order.
// Bound: by the tensor unit, 1.05 us a block of 16 rows, 1.3 of 64, 2 of 128, whatever the depth and the number of the warps that
// feed it (a product of 128 x 16 x 16 takes it 57 cycles).  204 x 4,096 x 1,024: 74 us by FMA (52% of their rate), so 27;
// 204 x 6,144 x 1,024 106 and 41; 204 x 1,024 x 3,072 57 and 21; one row of 1,024 x 3,072 21 and 16.  The head of 151,936 x 1,024 is
// slower at up to 8 rows (127 and 163), whose bits may not differ from those of 64 rows (596 and 232).
constexpr int BN = 128, BK = 64;
constexpr int PLANE_A = BN * BK * 2;                     // bytes of a part of W's rows
__device__ int dib_gemm_fp32_error_word;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// D[tmem] (+)= A[smem] * B[smem]^T, both operands K-major
__device__ __forceinline__ void tc_mma(unsigned tmem_d, unsigned long long desc_a, unsigned long long desc_b,
                                       unsigned idesc, unsigned accum) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accum), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void tc_ld(unsigned taddr, unsigned (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
__device__ __forceinline__ void tc_ld(unsigned taddr, unsigned (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
// K-major bfloat16 tile of rows of 128 bytes with the 128-byte swizzle: 8-row groups lie 1024 bytes apart
__device__ __forceinline__ unsigned long long smem_desc_sw128(unsigned addr) {
  return (unsigned long long)((addr & 0x3FFFFu) >> 4) | (unsigned long long)(1024u >> 4) << 32 | 1ull << 46 | 2ull << 61;
}
__host__ __device__ constexpr unsigned make_idesc(int m, int n) {      // float32 accumulator, bfloat16 operands, both K-major
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(m >> 4) << 24);
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_peer_smem(const float* local, unsigned rank) {
  unsigned remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}
// two float32 numbers, times 2^SCALE, as three pairs of bfloat16 numbers whose sums they are.  The third part of a number
// begins 16 bits below it: without the factor it would fall under bfloat16's smallest number, 2^-133, for numbers
// below 2^-109; with it every number that float32 holds, subnormal ones included, keeps all its bits.
constexpr int SCALE = 16;
__device__ __forceinline__ void take_apart(float x, float y, unsigned (&part)[3]) {
  float2 v = __fmul2_rn(make_float2(x, y), make_float2((float)(1 << SCALE), (float)(1 << SCALE)));
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
    part[i] = *reinterpret_cast<const unsigned*>(&h);
    if (i < 2)       // (exact)
      v = __ffma2_rn(make_float2(__uint_as_float(part[i] << 16), __uint_as_float(part[i] & 0xffff0000u)),
                     make_float2(-1.f, -1.f), v);
  }
}

// How a tile's four runs of k are divided (the order of the sums is the same).  RUNS: a CTA of the cluster takes a run.  PAIRS: two
// CTAs take two runs each, the first adds its two up, the second leaves both.  FOLD: one CTA takes all runs, one after
// the other (no cluster).  For grids that fill the GPU with less division.
constexpr int RUNS_OF_K = 4;         // (8 and 204 rows of 1,536, 512, us: two runs 8.2 and 10.1, four 5.7 and 9.5, eight 5.4 and 14.5)
enum Form { RUNS, PAIRS, FOLD };
constexpr int ctas_of(Form form) { return form == RUNS ? RUNS_OF_K : form == PAIRS ? 2 : 1; }

// TOK rows of A a CTA, NW warps that take operands apart, DEPTH blocks that a thread has asked for and not yet taken apart
template <int TOK, int NW, int DEPTH> struct Tc {
  static constexpr int PLANE_B = TOK * BK * 2;
  static constexpr int STAGE = 3 * (PLANE_A + PLANE_B);
  static constexpr int SUMS = TOK * BN * 4;              // the sums that a CTA leaves for its cluster
  static constexpr int SMEM = 2 * STAGE + 1024;          // (and the tiles' alignment)
  static_assert(2 * STAGE >= 2 * SUMS, "the sums of two runs fit the stages");
  static constexpr int CTAS = TOK <= 16 && NW == 8 && DEPTH == 1 ? 2 : 1;
  static constexpr int THREADS = NW * 32 + 32;           // (one more warp issues the products)
  static constexpr int TMEM_COLS = 2 * TOK < 32 ? 32 : 2 * TOK;
  static constexpr int STEP = 2 * NW;                    // rows between a thread's pieces of a block
  static constexpr int ROWS_A = BN / STEP, ROWS_B = TOK / STEP;     // its 16-byte pieces of the operands
};

// The results that a CTA's `odd` marks (columns c0 .. c_end - 1 of its tile), by FMA from the operands.  A row of A that holds
// a not-a-number has no other result; the others are sums over k by a warp for four columns, a chain a lane, the lanes by
// the butterfly.  (us, 4,096 x 1,024, finite / one not-a-number in each row / an infinity in one row: 1 row 10 / 16 / 25, 204 rows
// 27 / 54 / 38; all 204 rows with an infinity 295.  By the thread of each result 140, 3,730 and 156.)  A function of its own,
// called: in the kernel it takes registers from the loop (204 rows 28 -> 30 us).
__device__ __noinline__ void odd_results(const float* A, const float* W, float* out, unsigned char* odd, int m0, int n0,
                                         int c0, int c_end, int N, int K) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int c = c0 + warp; c < c_end; c += blockDim.x >> 5) {
    const unsigned bits = odd[c * (BN / 4) + lane];
    if (!__any_sync(0xffffffffu, bits != 0)) continue;
    const float* x = A + (size_t)(m0 + c) * K;
    bool nan = false;
#pragma unroll 8
    for (int k = lane; k < K; k += 32) nan = nan || x[k] != x[k];
    if (!__any_sync(0xffffffffu, nan)) continue;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (bits >> i & 1) out[(size_t)(m0 + c) * N + n0 + lane * 4 + i] = __int_as_float(0x7fffffff);
    odd[c * (BN / 4) + lane] = 0;
  }
  __syncthreads();
  for (int e = c0 * (BN / 4) + warp; e < c_end * (BN / 4); e += blockDim.x >> 5) {
    const unsigned bits = odd[e];
    if (bits == 0) continue;
    const int n = n0 + e % (BN / 4) * 4, m = m0 + e / (BN / 4);
    const float *x = A + (size_t)m * K, *y[4];
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = W + (size_t)min(n + i, N - 1) * K;
#pragma unroll 4
    for (int k = lane; k < K; k += 32) {
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i] = __fmaf_rn(x[k], y[i][k], s[i]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s[i] = warp_sum(s[i]);
      if (lane == i && (bits >> i & 1)) out[(size_t)m * N + n + i] = s[i];
    }
  }
}

template <int TOK, int NW, int DEPTH, bool VEC, Form FORM>
__global__ void __launch_bounds__((Tc<TOK, NW, DEPTH>::THREADS), (Tc<TOK, NW, DEPTH>::CTAS))
gemm_fp32_tc_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ out, int M, int N,
                    int K, int tile0) {
  using C = Tc<TOK, NW, DEPTH>;
  constexpr int PARTS = ctas_of(FORM), RUNS_EACH = RUNS_OF_K / PARTS;
  constexpr bool FOLDS = FORM != RUNS;
  constexpr int TC_THREADS = C::THREADS, WARPS = NW;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
  __shared__ unsigned long long done[2];                 // the products of the block in stage s have completed
  __shared__ unsigned tmem_slot;
  __shared__ unsigned char odd[TOK * (BN / 4)];          // of four neighbouring results: those that are no finite numbers
  pdl_trigger();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * TOK, n0 = (tile0 + blockIdx.x) * BN, part = blockIdx.z;
  const int n_end = min(N, n0 + BN);
  const int blocks = (K + BK - 1) / BK, per = (blocks + RUNS_OF_K - 1) / RUNS_OF_K;
  const int kb0 = part * RUNS_EACH * per, nkb = max(0, min(RUNS_EACH * per, blocks - kb0));
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&done[0])));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&done[1])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"((unsigned)C::TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  // a thread's pieces: 4 k from 4 (tid % 16) of rows tid / 16 + STEP i
  const int row = tid >> 4, c4 = tid & 15;
  float4 a[DEPTH][C::ROWS_A], b[DEPTH][C::ROWS_B];
  auto load = [&](const float* src, int r, int rows, int k) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows) {
      const float* at = src + (size_t)r * K + k;
      if (VEC) {
        if (k < K) v = *reinterpret_cast<const float4*>(at);
      } else {
        if (k < K) v.x = at[0];
        if (k + 1 < K) v.y = at[1];
        if (k + 2 < K) v.z = at[2];
        if (k + 3 < K) v.w = at[3];
      }
    }
    return v;
  };
  // A block that lies within K, rows on 16 bytes: a uniform base and a thread's offset, rows behind the last one's standing
  // in for it (their results go nowhere).  (Addresses and bounds apiece were half of the kernel's instructions.)
  const unsigned row_bytes = 4u * (unsigned)K, skip = C::STEP * row_bytes;
  const unsigned w_off = row * row_bytes + c4 * 16, w_last = (unsigned)(n_end - n0 - 1) * row_bytes + c4 * 16;
  const unsigned a_last = (unsigned)(min(TOK, M - m0) - 1) * row_bytes + c4 * 16;
  const bool near = VEC && K <= (1 << 22);               // (offsets within 32 bits)
  auto w_piece = [&](int kb, int i) { return load(W, n0 + row + C::STEP * i, n_end, (kb0 + kb) * BK + 4 * c4); };
  auto a_piece = [&](int kb, int i) { return load(A, m0 + row + C::STEP * i, M, (kb0 + kb) * BK + 4 * c4); };
  const bool mine = nkb > 0 && warp < WARPS;
  // W may have been computed just before (another activation): its first blocks are only brought into L2 ahead of the wait
#pragma unroll
  for (int d = 0; d < DEPTH; ++d)
#pragma unroll
    for (int i = 0; i < C::ROWS_A; ++i)
      if (mine && d < nkb && (c4 & 1) == 0 && n0 + row + C::STEP * i < n_end && (kb0 + d) * BK + 4 * c4 < K)
        prefetch_l2(W + (size_t)(n0 + row + C::STEP * i) * K + (kb0 + d) * BK + 4 * c4);
  pdl_wait(A, W);
  auto ask = [&](int kb, int d) {
    if (near && (kb0 + kb + 1) * BK <= K) {
      const char* wt = reinterpret_cast<const char*>(W + (size_t)n0 * K + (kb0 + kb) * BK);
      const char* at = reinterpret_cast<const char*>(A + (size_t)m0 * K + (kb0 + kb) * BK);
#pragma unroll
      for (int i = 0; i < C::ROWS_A; ++i) a[d][i] = *reinterpret_cast<const float4*>(wt + min(w_off + i * skip, w_last));
#pragma unroll
      for (int i = 0; i < C::ROWS_B; ++i) b[d][i] = *reinterpret_cast<const float4*>(at + min(w_off + i * skip, a_last));
      return;
    }
#pragma unroll
    for (int i = 0; i < C::ROWS_A; ++i) a[d][i] = w_piece(kb, i);
#pragma unroll
    for (int i = 0; i < C::ROWS_B; ++i) b[d][i] = a_piece(kb, i);
  };
#pragma unroll
  for (int d = 0; d < DEPTH; ++d)
    if (mine && d < nkb) ask(d, d);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = tmem_slot;
  // this thread's place in a part's tile: 8 bytes of row `row` (+ STEP i: the same swizzle)
  const int at = row * 128 + (((c4 >> 1) ^ (row & 7)) << 4) + (c4 & 1) * 8;
  constexpr unsigned idesc = make_idesc(BN, TOK);
  constexpr int HALF = TOK * 4 / NW, LD = HALF < 8 ? HALF : 8;   // a warp reads the rows 32 (warp % 4) .. of HALF columns
  float sum[HALF];
#pragma unroll
  for (int j = 0; j < HALF; ++j) sum[j] = 0.f;
  float total[FOLDS ? HALF : 1];       // of the runs before (PAIRS, second CTA: the first run, next to the second in `sum`)
  bool dead = false;                   // a wait has run out: no more waits, the launch is reported as failed
  auto add_block = [&](int kb) {
    if (!dead && !mbar_wait(&done[kb & 1], (kb >> 1) & 1)) dead = true;
    __syncwarp();
    tc_fence_after();
    const unsigned from = tmem + ((unsigned)((warp & 3) * 32) << 16) + (kb & 1) * TOK + (warp >> 2) * HALF;
#pragma unroll
    for (int j = 0; j < HALF; j += LD) {
      unsigned r[LD];
      tc_ld(from + j, r);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int e = 0; e < LD; ++e) sum[j + e] = __fadd_rn(sum[j + e], __uint_as_float(r[e]));
    }
    tc_fence_before();
    if (FOLDS && ((kb + 1) % per == 0 || kb + 1 == nkb) && !(FORM == PAIRS && part == 1 && kb >= per)) {
#pragma unroll
      for (int j = 0; j < HALF; ++j) {
        total[FOLDS ? j : 0] = kb < per ? sum[j] : __fadd_rn(total[FOLDS ? j : 0], sum[j]);
        sum[j] = 0.f;
      }
    }
  };
  if (warp == WARPS) {
    for (int kb = 0; kb < nkb; ++kb) {
      __syncthreads();                 // block kb's parts are there; the accumulator of block kb - 2 has been read
      if (lane == 0) {
        tc_fence_after();
        const unsigned stage = smem_u32(smem + (kb & 1) * C::STAGE);
        const unsigned long long da = smem_desc_sw128(stage), db = smem_desc_sw128(stage + 3 * PLANE_A);
        constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};      // the smallest products first
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
          for (int ks = 0; ks < BK / 16; ++ks)
            tc_mma(tmem + (kb & 1) * TOK, da + ((PA[p] * PLANE_A + ks * 32) >> 4), db + ((PB[p] * C::PLANE_B + ks * 32) >> 4),
                   idesc, p + ks > 0 ? 1u : 0u);
        tc_commit(&done[kb & 1]);
      }
      __syncwarp();
    }
  } else {
    for (int k0 = 0; k0 < nkb; k0 += DEPTH) {
#pragma unroll
      for (int d = 0; d < DEPTH; ++d) {
        const int kb = k0 + d;
        if (kb >= nkb) break;
        // the stage and the accumulator are free: the block before the last one has been added up
        unsigned char* stage = smem + (kb & 1) * C::STAGE;
        auto leave = [&](unsigned char* plane, int plane_bytes, const float4& v) {
          unsigned lo[3], hi[3];
          take_apart(v.x, v.y, lo);
          take_apart(v.z, v.w, hi);
#pragma unroll
          for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(plane + p * plane_bytes + at) = make_uint2(lo[p], hi[p]);
        };
#pragma unroll
        for (int i = 0; i < C::ROWS_A; ++i) leave(stage + i * C::STEP * 128, PLANE_A, a[d][i]);
#pragma unroll
        for (int i = 0; i < C::ROWS_B; ++i) leave(stage + 3 * PLANE_A + i * C::STEP * 128, C::PLANE_B, b[d][i]);
        if (kb + DEPTH < nkb) ask(kb + DEPTH, d);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (kb > 0) add_block(kb - 1);
      }
    }
    if (nkb > 0) add_block(nkb - 1);
  }
  if (dead) atomicExch(&dib_gemm_fp32_error_word, 1);
  // the runs' sums, in run order; a CTA of the cluster takes a share of the tile's columns (rows of A)
  __syncthreads();                     // (every product has completed: the stages are free)
  float* sums = reinterpret_cast<float*>(smem);          // [TOK][128 rows of W] (PAIRS: two of them)
  if (warp < WARPS) {
#pragma unroll
    for (int j = 0; j < HALF; ++j) {
      float* to = sums + ((warp >> 2) * HALF + j) * BN + (warp & 3) * 32 + lane;
      *to = FOLDS ? total[FOLDS ? j : 0] : sum[j];
      if (FORM == PAIRS) to[TOK * BN] = sum[j];
    }
  }
  if (PARTS > 1) cluster_sync_all();
  else __syncthreads();
  const int cols = min(TOK, M - m0), share = (cols + PARTS - 1) / PARTS;
  const int c_end = min(cols, (part + 1) * share);
  bool any = false;
  for (int e = part * share * (BN / 4) + tid; e < c_end * (BN / 4); e += TC_THREADS) {
    const int n = n0 + e % (BN / 4) * 4, m = m0 + e / (BN / 4);
    const float* p = sums + 4 * e;
    float4 v;
    if (PARTS > 1) {
      float4 run[PARTS + 1];
#pragma unroll
      for (int r = 0; r < PARTS; ++r) run[r] = ld_peer_smem(p, r);
      if (FORM == PAIRS) run[PARTS] = ld_peer_smem(p + TOK * BN, 1);
      v = run[0];
#pragma unroll
      for (int r = 1; r < (FORM == PAIRS ? PARTS + 1 : PARTS); ++r)
        v = make_float4(__fadd_rn(v.x, run[r].x), __fadd_rn(v.y, run[r].y), __fadd_rn(v.z, run[r].z), __fadd_rn(v.w, run[r].w));
    } else {
      v = *reinterpret_cast<const float4*>(p);
    }
    constexpr float DOWN = 1.0f / (1 << SCALE);
    const float o[4] = {v.x * DOWN * DOWN, v.y * DOWN * DOWN, v.z * DOWN * DOWN, v.w * DOWN * DOWN};
    unsigned bits = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)      // an operand or a sum that the scaled parts cannot hold
      if (n + i < n_end && !(fabsf(o[i]) <= 3.402823466e38f)) bits |= 1u << i;
    odd[e] = (unsigned char)bits;
    any = any || bits != 0;
    float* to = out + (size_t)m * N + n;
    if (n + 3 < n_end && (((uintptr_t)to) & 15) == 0) {
      *reinterpret_cast<float4*>(to) = make_float4(o[0], o[1], o[2], o[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (n + i < n_end) to[i] = o[i];
    }
  }
  __syncwarp();
  if (PARTS > 1) cluster_sync_all();   // nobody leaves while a peer may still read its sums
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)C::TMEM_COLS));
  if (__syncthreads_or(any)) odd_results(A, W, out, odd, m0, n0, part * share, c_end, N, K);
}

// Short sums (K below SHORT_K): one chain over all k in index order, as there is little to divide; the
// eight warps of a block take 16 x 32 outputs each of a tile of 64 x 64, from stages copied the same way.
// (204 rows: 768 x 192 9.7 us, 1,024 x 500 23 us; divided 5.9 and 12 us, but then the logits of a small
// model's ill-conditioned rows move by as much as they are off; 64 x 64 x 16 in order, as before: 21, 54 us.
// 512 lies between the sizes of such small models, whose bits stay as they were, and of real ones; it is no
// crossover: the divided form would be quicker, and nearer to 64 bits on average, below it too.)
constexpr int SHORT_K = 512, SH_B = 64, SH_BK = 32, SH_STAGES = 3, SH_LD = SH_BK + 4;
template <bool VEC>
__global__ void __launch_bounds__(THREADS)
gemm_fp32_short_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ out,
                       int M, int N, int K) {
  extern __shared__ __align__(16) float smem[];
  pdl_prologue(A, W);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r0 = (warp >> 1) * 16 + (lane >> 3), c0 = (warp & 1) * 32 + (lane & 7);      // + 4 i, + 8 j
  const int row_tiles = (M + SH_B - 1) / SH_B;
  const int m0 = (int)(blockIdx.x % row_tiles) * SH_B, n0 = (int)(blockIdx.x / row_tiles) * SH_B;
  const int steps = (K + SH_BK - 1) / SH_BK;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  auto fetch = [&](int s) {
    if (s < steps) {
      float* st = smem + (s % SH_STAGES) * 2 * SH_B * SH_LD;
      copy_rows<SH_B, SH_BK, SH_LD, VEC>(st, A, m0, M, s * SH_BK, K);
      copy_rows<SH_B, SH_BK, SH_LD, VEC>(st + SH_B * SH_LD, W, n0, N, s * SH_BK, K);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < SH_STAGES - 1; ++s) fetch(s);
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(SH_STAGES - 2) : "memory");
    __syncthreads();                 // stage s is there for all; stage s - 1 has been read by all
    fetch(s + SH_STAGES - 1);
    const float* sa = smem + (s % SH_STAGES) * 2 * SH_B * SH_LD + r0 * SH_LD;
    const float* sw = smem + (s % SH_STAGES) * 2 * SH_B * SH_LD + (SH_B + c0) * SH_LD;
#pragma unroll
    for (int k = 0; k < SH_BK; k += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = *reinterpret_cast<const float4*>(sa + 4 * i * SH_LD + k);
        b[i] = *reinterpret_cast<const float4*>(sw + 8 * i * SH_LD + k);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
          acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
          acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
        }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = m0 + r0 + 4 * i, c = n0 + c0 + 8 * j;
      if (r < M && c < N) out[(size_t)r * N + c] = acc[i][j];
    }
}

template <int TOK, int NW, int DEPTH, bool VEC, Form FORM>
int launch_form(const float* A, const float* W, float* out, int M, int N, int K, int tile0, int tiles, cudaStream_t st) {
  using C = Tc<TOK, NW, DEPTH>;
  static DeviceOnce once;
  if (!once.done()) {
    if (cudaFuncSetAttribute(gemm_fp32_tc_kernel<TOK, NW, DEPTH, VEC, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) !=
        cudaSuccess) {
      cudaGetLastError();
      return DIB_LAUNCH_FAILED;
    }
    once.mark();
  }
  constexpr int parts = ctas_of(FORM);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles, ceil_div_host(M, TOK), parts);
  cfg.blockDim = dim3(C::THREADS);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = (unsigned)parts;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dib_pdl_enabled() ? 2 : 1;
  cudaLaunchKernelEx(&cfg, gemm_fp32_tc_kernel<TOK, NW, DEPTH, VEC, FORM>, A, W, out, M, N, K, tile0);
  DIB_CHECK_LAUNCH();
  return DIB_OK;
}
template <bool VEC>
int launch_short(const float* A, const float* W, float* out, int M, int N, int K, cudaStream_t st) {
  constexpr int smem = 4 * SH_STAGES * 2 * SH_B * SH_LD;           // 55 KB
  static DeviceOnce once;
  if (!once.done()) {
    if (cudaFuncSetAttribute(gemm_fp32_short_kernel<VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
      cudaGetLastError();
      return DIB_LAUNCH_FAILED;
    }
    once.mark();
  }
  const long long blocks = (long long)ceil_div_host(M, SH_B) * ceil_div_host(N, SH_B);
  if (blocks > 0x7fffffffll) return DIB_BAD_SIZE;
  dib_launch(gemm_fp32_short_kernel<VEC>, dim3((unsigned)blocks), dim3(THREADS), smem, st, A, W, out, M, N, K);
  DIB_CHECK_LAUNCH();
  return DIB_OK;
}
// 16-byte copies want rows that start on 16 bytes
bool takes_vectors(const float* A, const float* W, int K) { return K % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0; }
template <int TOK, int NW, int DEPTH, Form FORM>
int launch(const float* A, const float* W, float* out, int M, int N, int K, cudaStream_t st, int tile0 = 0, int tiles = -1) {
  if (tiles < 0) tiles = ceil_div_host(N, BN);
  return takes_vectors(A, W, K) ? launch_form<TOK, NW, DEPTH, true, FORM>(A, W, out, M, N, K, tile0, tiles, st)
                                : launch_form<TOK, NW, DEPTH, false, FORM>(A, W, out, M, N, K, tile0, tiles, st);
}

// Which tile and form: the one whose last wave of CTAs is done first.  A CTA takes `fixed` us (launch, first operands, the
// runs' sum) and `block` us for each of its blocks of 64 k; `at_once` CTAs fit the GPU.  Fitted to single products with weights from
// memory, us (tile rows and form: measured): 1 row of 1,024, 3,072 and 1,024, 2,048 (16 RUNS) 16.1, 12.1; 17 rows (32 RUNS) 18.1, 13.5;
// 204 rows (64 RUNS) 20.6, 15.5; 204 x 4,096 x 1,024 (64 FOLD, 128 RUNS, 64 RUNS) 26, 27, 41; 500 x 4,096 x 1,024 (128 FOLD, 128
// RUNS) 44, 54; the head of 151,936 x 1,024 at 8, 17, 64 and 204 rows (16, 32, 64, 128 FOLD) 163, 194, 232, 776, where the RUNS took
// 209, 335, 387 and 1,030; 17, 64 and 46 rows of 6,144, 1,024, 1,024 and 512 (32, 64, 64 PAIRS; RUNS have two waves there) 14.5, 18.2, 11.5
// against 18.3, 20.5, 13.3.  Up to 16 rows two CTAs share an SM with a block asked for ahead, or one has it with two:
// 8 rows of 6,144, 1,024 (192 CTAs) 13.3 / 17.3, of 4,096, 1,024 (128) 12.4 / 9.2.  What waits is the tensor unit: a product of 128 x 16 x 16
// takes it 57 cycles as one of 128 x 32 x 16 nearly does, 24 of them a block.
struct Choice {
  int form = -1;
  float time = 1e30f;
  void consider(int id, float t) {
    if (t < time) form = id, time = t;
  }
};
struct Sizes {
  int M, N, K;
  int blocks() const { return ceil_div_host(K, BK); }
  long long tiles(int tok) const { return (long long)ceil_div_host(N, BN) * ceil_div_host(M, tok); }
  bool fits(int tok) const { return ceil_div_host(M, tok) <= 65535; }
  float divided(Form form, int tok, int at_once, float fixed, float block) const {
    if (!fits(tok)) return 1e30f;
    const int per = (blocks() + RUNS_OF_K - 1) / RUNS_OF_K * (RUNS_OF_K / ctas_of(form));
    return (float)((tiles(tok) * ctas_of(form) + at_once - 1) / at_once) * (fixed + block * per);
  }
  // FOLD: a last wave of a few tiles (the head of 151,936: 1,187 tiles, 8 waves of 148 and 3) is a grid of RUNS of its own
  int tail(int tok, int at_once) const {
    const long long all = tiles(tok), left = all % at_once;
    return M <= tok && all > at_once && left * RUNS_OF_K <= 148 ? (int)left : 0;
  }
  float fold(int tok, int at_once, float fixed, float block) const {
    if (!fits(tok)) return 1e30f;
    const long long all = tiles(tok);
    const int left = tail(tok, at_once);
    return (float)((all - left + at_once - 1) / at_once) * (fixed + block * blocks()) + (left > 0 ? 6.f : 0.f);
  }
};
template <int TOK, int NW, int DEPTH, int RUNS_NW, int RUNS_DEPTH>
int launch_fold(const float* A, const float* W, float* out, const Sizes& z, int at_once, cudaStream_t st) {
  const int left = z.tail(TOK, at_once), tiles = ceil_div_host(z.N, BN);
  const int status = launch<TOK, NW, DEPTH, FOLD>(A, W, out, z.M, z.N, z.K, st, 0, tiles - left);
  if (status != DIB_OK || left == 0) return status;
  return launch<TOK, RUNS_NW, RUNS_DEPTH, RUNS>(A, W, out, z.M, z.N, z.K, st, tiles - left, left);
}

}  // namespace

// 0, or the code of a wait that ran out in a launch since the word was cleared (-1: it could not be read)
extern "C" int dib_gemm_fp32_status() {
  int v = 0;
  return cudaMemcpyFromSymbol(&v, dib_gemm_fp32_error_word, sizeof(int)) == cudaSuccess ? v : -1;
}
extern "C" int dib_gemm_fp32_status_clear() {
  const int zero = 0;
  return cudaMemcpyToSymbol(dib_gemm_fp32_error_word, &zero, sizeof(int)) == cudaSuccess ? 0 : -1;
}
extern "C" int dib_gemm_fp32(const float* A, const float* W, float* out, int M, int N, int K,
                             cudaStream_t st) {
  if (M == 0 || N == 0) return DIB_OK;
  if (K <= 0) return DIB_BAD_SIZE;
  if (ceil_div_host(M, 64) > 65535) return DIB_BAD_SIZE;
  if (K < SHORT_K)
    return takes_vectors(A, W, K) ? launch_short<true>(A, W, out, M, N, K, st) : launch_short<false>(A, W, out, M, N, K, st);
  const Sizes z{M, N, K};
  Choice best;
  if (M <= 16) {
    best.consider(0, z.divided(RUNS, 16, 148, 3.8f, 1.04f));
    best.consider(1, z.divided(RUNS, 16, 296, 3.5f, 2.4f));
    best.consider(2, z.fold(16, 296, 3.5f, z.tiles(16) > 148 ? 2.1f : 1.4f));
  }
  best.consider(3, z.divided(RUNS, 32, 148, 4.6f, 1.13f));
  best.consider(4, z.fold(32, 148, 4.5f, 1.12f));
  best.consider(5, z.divided(RUNS, 64, 148, 5.3f, 1.25f));
  best.consider(6, z.fold(64, 148, 5.1f, 1.32f));
  best.consider(7, z.divided(RUNS, 128, 148, 4.9f, 1.98f));
  best.consider(8, z.fold(128, 148, 10.5f, 2.07f));
  if (M <= 16) best.consider(9, z.divided(PAIRS, 16, 148, 4.6f, 1.08f));
  best.consider(10, z.divided(PAIRS, 32, 148, 5.2f, 1.17f));
  best.consider(11, z.divided(PAIRS, 64, 148, 5.0f, 1.62f));
  best.consider(12, z.divided(PAIRS, 128, 148, 8.2f, 2.2f));
  switch (best.form) {
    case 0: return launch<16, 8, 2, RUNS>(A, W, out, M, N, K, st);
    case 1: return launch<16, 8, 1, RUNS>(A, W, out, M, N, K, st);
    case 2: return launch_fold<16, 8, 1, 8, 2>(A, W, out, z, 296, st);
    case 3: return launch<32, 8, 1, RUNS>(A, W, out, M, N, K, st);
    case 4: return launch_fold<32, 8, 2, 8, 1>(A, W, out, z, 148, st);
    case 5: return launch<64, 16, 1, RUNS>(A, W, out, M, N, K, st);
    case 6: return launch_fold<64, 8, 1, 16, 1>(A, W, out, z, 148, st);
    case 7: return launch<128, 16, 1, RUNS>(A, W, out, M, N, K, st);
    case 8: return launch_fold<128, 16, 1, 16, 1>(A, W, out, z, 148, st);
    case 9: return launch<16, 8, 2, PAIRS>(A, W, out, M, N, K, st);
    case 10: return launch<32, 8, 1, PAIRS>(A, W, out, M, N, K, st);
    case 11: return launch<64, 16, 1, PAIRS>(A, W, out, M, N, K, st);
    default: return launch<128, 16, 1, PAIRS>(A, W, out, M, N, K, st);
  }
}

// True float32 matrix product on the CUDA cores: C[M,N] = A[M,K] * W[N,K]^T.
//
// This is the matrix product of the 32-bit path: plain FMA, no tensor cores and
// no reduced-precision mode.  From K = 512 on an output element is eight partial sums: k
// belongs to partial (k / 4) % 8, each partial adds its k in index order, and the partials
// are added one after the other.  Below, it is one chain over k in index order
// (gemm_fp32_short_kernel).  The order is a function of K alone, whatever the tile, so a
// row's result does not depend on M: the same token gives the same bits in any batch.
// (Distance from 64-bit sums at K = 1024 .. 3072: 2.1e-7 .. 3.6e-7 of the norm.  The logits
// of 204 rows through 28 layers came to 9.1e-7, against 2.1e-6 with one chain over all k.)
//
// Both operands lie k-contiguous, and stay so in shared memory (copied 16 bytes at a
// time, two or three stages ahead).  The eight warps of a block share one output tile
// and divide k, warp w taking the partial w, so that even a tile of few outputs keeps
// an SM's four schedulers busy with large thread tiles.  A thread reads four k of a row
// with one 16-byte load: 16 loads for 256 FMA at 8 x 8 outputs a thread.
// Bound: shared-memory reads and FMA issue about equally (8 x 8 outputs a thread, two
// blocks an SM: 1000 x 4096 x 1024 in 262 us, 52% of the FMA rate; paired FMA with
// even and odd k in one instruction needs twice the accumulators, one block an SM:
// 299 us); the weights' bytes for a few rows (8 x 151936 x 1024: 136 us, 4.6 TB/s).
#include "common.cuh"

namespace {

constexpr int WARPS = 8;             // k is divided over them: part of the order above
constexpr int THREADS = WARPS * 32;

template <int BM_, int BN_, int TM_, int TN_, int BK_, int STAGES_, int CTAS_>
struct Tile {
  static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, BK = BK_, STAGES = STAGES_, CTAS = CTAS_;
  static constexpr int LM = BM / TM, LN = BN / TN;         // lanes over rows and columns
  static constexpr int LD = BK + 4;                        // row of a stage: 8 rows start in 8 different bank groups
  static constexpr int LDR = BN + 4;                       // row of a warp's sums
  static constexpr int STAGE = (BM + BN) * LD;             // floats
  static constexpr int SMEM = 4 * (STAGES * STAGE > WARPS * BM * LDR ? STAGES * STAGE : WARPS * BM * LDR);
  static_assert(LM * LN == 32 && BK % (4 * WARPS) == 0, "a warp holds the tile; every warp has k in every stage");
};

// rows r0 .. r0 + ROWS - 1 (below `rows`), k0 .. k0 + BK - 1 (below K) of a [rows, K] matrix; zeros elsewhere
template <int ROWS, int BK, int LD, bool VEC>
__device__ __forceinline__ void copy_rows(float* dst, const float* __restrict__ src, int r0, int rows, int k0, int K) {
  constexpr int E = VEC ? 4 : 1, PER = BK / E;             // elements a copy, copies a row
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

template <typename C, bool VEC>
__global__ void __launch_bounds__(THREADS, C::CTAS)
gemm_fp32_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ out,
                 int M, int N, int K) {
  extern __shared__ __align__(16) float smem[];
  pdl_prologue(A, W);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ty = lane / C::LN, tx = lane % C::LN;
  // row tiles lie next to one another: blocks that run together read the same weights
  const int row_tiles = (M + C::BM - 1) / C::BM;
  const int m0 = (int)(blockIdx.x % row_tiles) * C::BM, n0 = (int)(blockIdx.x / row_tiles) * C::BN;
  const int steps = (K + C::BK - 1) / C::BK;

  float acc[C::TM][C::TN];
#pragma unroll
  for (int i = 0; i < C::TM; ++i)
#pragma unroll
    for (int j = 0; j < C::TN; ++j) acc[i][j] = 0.f;

  auto fetch = [&](int s) {
    if (s < steps) {
      float* st = smem + (s % C::STAGES) * C::STAGE;
      copy_rows<C::BM, C::BK, C::LD, VEC>(st, A, m0, M, s * C::BK, K);
      copy_rows<C::BN, C::BK, C::LD, VEC>(st + C::BM * C::LD, W, n0, N, s * C::BK, K);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < C::STAGES - 1; ++s) fetch(s);

  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(C::STAGES - 2) : "memory");
    __syncthreads();                 // stage s is there for all; stage s - 1 has been read by all
    fetch(s + C::STAGES - 1);
    const float* sa = smem + (s % C::STAGES) * C::STAGE;
    const float* sw = sa + C::BM * C::LD;
#pragma unroll
    for (int k = 0; k < C::BK; k += 4 * WARPS) {
      const int at = k + warp * 4;
      float4 a[C::TM];
#pragma unroll
      for (int i = 0; i < C::TM; ++i)
        a[i] = *reinterpret_cast<const float4*>(sa + (i * C::LM + ty) * C::LD + at);
#pragma unroll
      for (int j = 0; j < C::TN; ++j) {
        const float4 b = *reinterpret_cast<const float4*>(sw + (j * C::LN + tx) * C::LD + at);
#pragma unroll
        for (int i = 0; i < C::TM; ++i) acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
#pragma unroll
        for (int i = 0; i < C::TM; ++i) acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
#pragma unroll
        for (int i = 0; i < C::TM; ++i) acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
#pragma unroll
        for (int i = 0; i < C::TM; ++i) acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // the warps' sums meet in shared memory and are added in the warps' order
  float* mine = smem + warp * C::BM * C::LDR;
#pragma unroll
  for (int i = 0; i < C::TM; ++i)
#pragma unroll
    for (int j = 0; j < C::TN; ++j) {
      mine[(i * C::LM + ty) * C::LDR + j * C::LN + tx] = acc[i][j];
    }
  __syncthreads();
  for (int o = threadIdx.x; o < C::BM * C::BN; o += THREADS) {
    const int r = o / C::BN, c = o % C::BN;
    const float* p = smem + r * C::LDR + c;
    float v = p[0];
#pragma unroll
    for (int w = 1; w < WARPS; ++w) v = __fadd_rn(v, p[w * C::BM * C::LDR]);
    if (m0 + r < M && n0 + c < N) out[(size_t)(m0 + r) * N + n0 + c] = v;
  }
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

template <typename C, bool VEC>
int launch_vec(const float* A, const float* W, float* out, int M, int N, int K, cudaStream_t st) {
  static DeviceOnce once;
  if (!once.done()) {
    if (cudaFuncSetAttribute(gemm_fp32_kernel<C, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess) {
      cudaGetLastError();
      return DIB_LAUNCH_FAILED;
    }
    once.mark();
  }
  const long long blocks = (long long)ceil_div_host(M, C::BM) * ceil_div_host(N, C::BN);
  if (blocks > 0x7fffffffll) return DIB_BAD_SIZE;
  dib_launch(gemm_fp32_kernel<C, VEC>, dim3((unsigned)blocks), dim3(THREADS), C::SMEM, st, A, W, out, M, N, K);
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
template <typename C>
int launch(const float* A, const float* W, float* out, int M, int N, int K, cudaStream_t st) {
  return takes_vectors(A, W, K) ? launch_vec<C, true>(A, W, out, M, N, K, st) : launch_vec<C, false>(A, W, out, M, N, K, st);
}

// The tiles, by rows and columns.  The choice: the tile whose fullest SM is done first.  With
// q tiles on it that takes max(alone, q * busy): `alone` is one tile by itself (latency), `busy`
// what a tile adds on an SM that has several; measured per 1024 k, in us.  (M = 64, N = 4096:
// 8 x 32 38.9, 16 x 32 32.8, 32 x 32 28.7, 64 x 32 30.7 us a call; M = 212, N = 1024, K = 2048:
// 16 x 32 57, 32 x 32 49, 64 x 32 51; a step of
// 204 rows of a 28-layer model: 38.8 ms, against 67.1 ms with tiles of 64 x 64 x 16, one in flight.)  The rule
// counts a B200's 148 SMs; every tile gives the same bits.
using T64 = Tile<64, 32, 8, 8, 32, 3, 2>;
using T32 = Tile<32, 32, 8, 4, 64, 3, 2>;
using T16 = Tile<16, 32, 4, 4, 64, 3, 3>;
using T8w = Tile<8, 64, 4, 4, 64, 4, 2>;
using T8 = Tile<8, 32, 2, 4, 64, 4, 3>;

template <typename C> float estimate(int M, int N, float alone, float busy) {
  const long long tiles = (long long)ceil_div_host(M, C::BM) * ceil_div_host(N, C::BN);
  const float q = (float)((tiles + 147) / 148);
  return q * busy > alone ? q * busy : alone;
}

}  // namespace

extern "C" int dib_gemm_fp32(const float* A, const float* W, float* out, int M, int N, int K,
                             cudaStream_t st) {
  if (M == 0 || N == 0) return DIB_OK;
  if (K <= 0) return DIB_BAD_SIZE;
  if (ceil_div_host(M, 64) > 65535) return DIB_BAD_SIZE;
  if (K < SHORT_K)
    return takes_vectors(A, W, K) ? launch_short<true>(A, W, out, M, N, K, st) : launch_short<false>(A, W, out, M, N, K, st);
  const float cost[5] = {estimate<T8>(M, N, 7.f, 4.3f), estimate<T8w>(M, N, 10.f, 7.2f), estimate<T16>(M, N, 8.f, 6.3f),
                         estimate<T32>(M, N, 13.f, 11.f), estimate<T64>(M, N, 22.f, 18.7f)};
  int best = 0;
  for (int i = 1; i < 5; ++i)
    if (cost[i] < cost[best]) best = i;
  switch (best) {
    case 0: return launch<T8>(A, W, out, M, N, K, st);
    case 1: return launch<T8w>(A, W, out, M, N, K, st);
    case 2: return launch<T16>(A, W, out, M, N, K, st);
    case 3: return launch<T32>(A, W, out, M, N, K, st);
    default: return launch<T64>(A, W, out, M, N, K, st);
  }
}

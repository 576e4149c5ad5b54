// Generic paged attention: float32 arithmetic throughout (expf, not the fast
// intrinsic), any head_dim up to 256, any number of heads and groups, any page size,
// optional window.  It is the attention of the 32-bit path, and the fallback of the
// bfloat16 path for head sizes the tensor-core kernels refuse.
//
// Every token of the step is one query: token t belongs to sequence
// token_seq[t], stands at absolute position positions[t] and sees the keys
// max(0, pos-window+1) .. pos of its sequence, all read from the paged cache
// through the sequence's row of the block table (this step's keys were written
// before the launch).  Keys are visited in tiles of 32 anchored at position 0,
// so the order of the reduction for a query depends on its position alone:
// the same token gives the same bits however the prompt was cut into steps,
// whatever else is in the batch and whichever pages hold its keys.
//
// A block has 16 neighbouring (token, head of the group) queries of one key-value head,
// or those of them that belong to one sequence: block (x, y) takes the y-th run of equal
// sequences among the 16 and ends at once where there is none.  So the tile of keys and
// values is read into shared memory once (the next tile's copies are in flight meanwhile)
// for up to 16 queries, two a warp: a prompt's queries share it, a decoding token has
// a block of its own.  Bound: a warp's chain through a tile (dot products, two reductions over the
// lanes, values), so the two queries of a warp go through it side by side and there are eight warps.  (16 heads
// of 128, us a layer, with four warps of four queries one after the other / so: 200 tokens behind
// 100 63 / 45, 300 behind 300 beside 8 of 1,000 keys 182 / 156, one token of 600 keys 49 / 44.  With three buffers of two tiles under way
// the same or slower: 45, 160, 45, and fewer blocks an SM: bfloat16 heads of 192, 1,000 tokens 939 / 659.)
//
// Cache layout of a layer: [num_pages, 2, num_kv_heads, page_size, head_dim].
#include "common.cuh"

#include <type_traits>

namespace {

constexpr int MAX_D = 256;
constexpr int ITEMS = 16;                      // queries a block
constexpr int KEYS = 32, BUFS = 2;             // keys of a tile; tiles in shared memory (one under way)
constexpr float NEG_BIG = -1e30f;

// floats between rows of a tile: rows padded to whole vectors, an odd number of vectors apart (the
// lanes' rows then start in different banks)
__host__ __device__ __forceinline__ int row_stride(int D) {
  const int v = (D + 3) / 4;
  return 4 * (v + 1 + (v & 1));
}
__host__ __device__ __forceinline__ int smem_floats(int D) {
  return 2 * BUFS * KEYS * row_stride(D) + ITEMS * row_stride(D) + ITEMS * KEYS;
}

// dot products of the lane's key with N queries, d in index order
template <int N, int NQ>
__device__ __forceinline__ void dots(const float* krow, const float* q, int ld, int vecs, float (&s)[NQ]) {
#pragma unroll
  for (int i = 0; i < N; ++i) s[i] = 0.f;
#pragma unroll 4
  for (int v = 0; v < vecs; ++v) {
    const float4 k = *reinterpret_cast<const float4*>(krow + 4 * v);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float4 x = *reinterpret_cast<const float4*>(q + i * ld + 4 * v);
      s[i] = fmaf(x.x, k.x, s[i]);
      s[i] = fmaf(x.y, k.y, s[i]);
      s[i] = fmaf(x.z, k.z, s[i]);
      s[i] = fmaf(x.w, k.w, s[i]);
    }
  }
}

// NV: vectors of four dimensions a lane owns (1: D <= 128).  ASYNC: float32 rows on 16 bytes.
template <typename T, int NV, bool ASYNC, int WARPS, int BLOCKS>
__global__ void __launch_bounds__(WARPS * 32, BLOCKS)
paged_attention_generic_kernel(const T* __restrict__ q, T* __restrict__ out,
                               const T* __restrict__ kv_cache,
                               const int* __restrict__ block_table, int max_blocks,
                               const int* __restrict__ token_seq,
                               const int* __restrict__ positions, int T_tokens, int Hq, int Hkv,
                               int D, int page_size, float scale, int window) {
  constexpr int THREADS = WARPS * 32, NQ = ITEMS / WARPS;      // (queries a warp)
  extern __shared__ __align__(16) float smem[];
  pdl_prologue(q, kv_cache, block_table, token_seq, positions);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = Hq / Hkv, kvh = blockIdx.x % Hkv;
  const long long item0 = (long long)(blockIdx.x / Hkv) * ITEMS, items = (long long)T_tokens * group;

  // the block's run of queries
  const long long item = item0 + lane;
  const bool there = lane < ITEMS && item < items;
  const int my_t = there ? (int)(item / group) : 0;
  const int my_seq = there ? token_seq[my_t] : -1;
  const int my_pos = there ? positions[my_t] : -1;
  const int before = __shfl_up_sync(0xffffffffu, my_seq, 1);
  const unsigned starts = __ballot_sync(0xffffffffu, there && (lane == 0 || my_seq != before));
  const int run = __popc(starts & (0xffffffffu >> (31 - lane))) - 1;
  const unsigned mine = __ballot_sync(0xffffffffu, there && run == (int)blockIdx.y);
  if (mine == 0u) return;                                // (the same for the whole block)
  const int lane0 = __ffs(mine) - 1, count = __popc(mine);
  const int seq = __shfl_sync(0xffffffffu, my_seq, lane0);
  const bool in_run = (mine >> lane) & 1u;
  const int my_first = window > 0 && my_pos - window + 1 > 0 ? my_pos - window + 1 : 0;
  int lo = in_run ? my_first : 0x7fffffff, hi = in_run ? my_pos : -1;   // keys the run sees
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }

  const int ld = row_stride(D), vecs = (D + 3) / 4;
  float* sk = smem;                                      // [BUFS][KEYS][ld]
  float* sv = sk + BUFS * KEYS * ld;
  float* sq = sv + BUFS * KEYS * ld + warp * NQ * ld;    // this warp's queries
  float* sp = smem + 2 * BUFS * KEYS * ld + ITEMS * ld + warp * NQ * KEYS;

  // queries number warp, warp + WARPS, ... of the run are this warp's
  int nq = 0, first[NQ], pos[NQ];
  long long row[NQ];
#pragma unroll
  for (int i = 0; i < NQ; ++i) {
    const int n = warp + i * WARPS;
    const int src = lane0 + (n < count ? n : 0);
    first[i] = __shfl_sync(0xffffffffu, my_first, src);
    pos[i] = __shfl_sync(0xffffffffu, my_pos, src);
    const int t = __shfl_sync(0xffffffffu, my_t, src);
    row[i] = ((long long)t * Hq + kvh * group + (int)((item0 + src) % group)) * D;
    if (n < count) nq = i + 1;
    for (int d = lane; d < 4 * vecs; d += 32)
      sq[i * ld + d] = n < count && d < D ? Elem<T>::load(q + row[i] + d) : 0.f;
  }

  const int* bt = block_table + (size_t)seq * max_blocks;
  const size_t head_stride = (size_t)page_size * D;          // one head inside a page
  const size_t kv_stride = (size_t)Hkv * head_stride;        // keys -> values inside a page
  const size_t page_stride = 2 * kv_stride;
  const int row0 = threadIdx.x / vecs, col0 = threadIdx.x % vecs;
  const int row_step = THREADS / vecs, col_step = THREADS % vecs;

  // the lane's page of a tile, asked for a tile ahead of its copies
  auto page_of = [&](int k0) {
    const int key = k0 + lane;
    return key >= lo && key <= hi ? bt[key / page_size] : -1;
  };
  auto fetch = [&](int k0, int buf, int page) {
    long long off = -1;                                  // of the lane's key; rows nobody sees become zeros
    if (page >= 0)
      off = (long long)((size_t)page * page_stride + (size_t)kvh * head_stride + (size_t)((k0 + lane) % page_size) * D);
    float* dk = sk + buf * KEYS * ld;
    float* dv = sv + buf * KEYS * ld;
    int r = row0, c = col0;
    for (int i = threadIdx.x; i < KEYS * vecs; i += THREADS) {   // (whole warps: KEYS * vecs is a multiple of 32)
      const long long o = __shfl_sync(0xffffffffu, off, r);
      if constexpr (ASYNC) {
        const T* src = kv_cache + (o < 0 ? 0 : o + 4 * c);
        const unsigned n = o < 0 ? 0u : 16u;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::
                         "r"((unsigned)__cvta_generic_to_shared(dk + r * ld + 4 * c)), "l"(src), "r"(n) : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::
                         "r"((unsigned)__cvta_generic_to_shared(dv + r * ld + 4 * c)), "l"(o < 0 ? src : src + kv_stride),
                         "r"(n) : "memory");
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int d = 4 * c + e;
          const bool in = o >= 0 && d < D;
          dk[r * ld + d] = in ? Elem<T>::load(kv_cache + o + d) : 0.f;
          dv[r * ld + d] = in ? Elem<T>::load(kv_cache + o + kv_stride + d) : 0.f;
        }
      }
      r += row_step;
      c += col_step;
      if (c >= vecs) {
        c -= vecs;
        ++r;
      }
    }
    if constexpr (ASYNC) asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float m[NQ], l[NQ];
  float4 acc[NQ][NV];
#pragma unroll
  for (int i = 0; i < NQ; ++i) {
    m[i] = NEG_BIG;
    l[i] = 0.f;
#pragma unroll
    for (int n = 0; n < NV; ++n) acc[i][n] = make_float4(0.f, 0.f, 0.f, 0.f);
  }

  const int begin = lo / KEYS * KEYS;
  const int page0 = page_of(begin);
  int page = page_of(begin + KEYS);
  fetch(begin, 0, page0);
  int buf = 0;
  for (int k0 = begin; k0 <= hi; k0 += KEYS, buf ^= 1) {
    if constexpr (ASYNC) asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                     // tile k0 is there; the one before has been read
    if (k0 + KEYS <= hi) {
      const int now = page;
      page = page_of(k0 + 2 * KEYS);
      fetch(k0 + KEYS, buf ^ 1, now);
    }
    if (nq == 0) continue;
    const float* krow = sk + (buf * KEYS + lane) * ld;
    float s[NQ];
    if (nq == 1) dots<1>(krow, sq, ld, vecs, s);
    else dots<NQ>(krow, sq, ld, vecs, s);
    const int key = k0 + lane;
    bool whole = true;                                   // every query of the warp sees the whole tile
    // the queries side by side: one that sees none of the tile keeps its maximum and is scaled by one
    float x[NQ], p[NQ], alpha[NQ];
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
      const bool live = i < nq;
      whole = whole && (!live || (first[i] <= k0 && pos[i] >= k0 + KEYS - 1));
      x[i] = live && key >= first[i] && key <= pos[i] ? s[i] * scale : NEG_BIG;
      p[i] = x[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < NQ; ++i) p[i] = fmaxf(p[i], __shfl_xor_sync(0xffffffffu, p[i], o));
    bool sees[NQ];
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
      sees[i] = i < nq && first[i] <= k0 + KEYS - 1 && pos[i] >= k0;
      const float m_new = fmaxf(m[i], p[i]);             // (the tile holds a visible key where the query sees it)
      p[i] = sees[i] && key >= first[i] && key <= pos[i] ? expf(x[i] - m_new) : 0.f;
      alpha[i] = sees[i] ? expf(m[i] - m_new) : 1.f;
      if (sees[i]) m[i] = m_new;
      if (i < nq) sp[i * KEYS + lane] = p[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < NQ; ++i) p[i] += __shfl_xor_sync(0xffffffffu, p[i], o);
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
      if (!sees[i]) continue;
      l[i] = fmaf(l[i], alpha[i], p[i]);
#pragma unroll
      for (int n = 0; n < NV; ++n) {
        acc[i][n].x *= alpha[i];
        acc[i][n].y *= alpha[i];
        acc[i][n].z *= alpha[i];
        acc[i][n].w *= alpha[i];
      }
    }
    __syncwarp();
    // P.V: keys in order, a lane owns the dimensions 4 * lane ..
    const float* vt = sv + buf * KEYS * ld + 4 * lane;
    auto add = [&](int i, float p, const float4 (&v)[NV]) {
#pragma unroll
      for (int n = 0; n < NV; ++n) {
        acc[i][n].x = fmaf(p, v[n].x, acc[i][n].x);
        acc[i][n].y = fmaf(p, v[n].y, acc[i][n].y);
        acc[i][n].z = fmaf(p, v[n].z, acc[i][n].z);
        acc[i][n].w = fmaf(p, v[n].w, acc[i][n].w);
      }
    };
    auto value = [&](int j, float4 (&v)[NV]) {
#pragma unroll
      for (int n = 0; n < NV; ++n)
        v[n] = lane + 32 * n < vecs ? *reinterpret_cast<const float4*>(vt + j * ld + 128 * n)
                                    : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    if (whole) {
#pragma unroll 2
      for (int j = 0; j < KEYS; j += 4) {
        float4 v0[NV], v1[NV], v2[NV], v3[NV];
        value(j, v0);
        value(j + 1, v1);
        value(j + 2, v2);
        value(j + 3, v3);
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
          if (i >= nq) break;
          const float4 p = *reinterpret_cast<const float4*>(sp + i * KEYS + j);
          add(i, p.x, v0);
          add(i, p.y, v1);
          add(i, p.z, v2);
          add(i, p.w, v3);
        }
      }
    } else {
      const int j1 = min(KEYS - 1, hi - k0);
      for (int j = 0; j <= j1; ++j) {
        float4 v[NV];
        value(j, v);
#pragma unroll
        for (int i = 0; i < NQ; ++i)      // (a key that a query does not see adds nothing, not even 0 times its value)
          if (i < nq && k0 + j >= first[i] && k0 + j <= pos[i]) add(i, sp[i * KEYS + j], v);
      }
    }
    __syncwarp();                                        // sp is written again in the next tile
  }
#pragma unroll
  for (int i = 0; i < NQ; ++i) {
    if (i >= nq) break;
    const float inv = 1.0f / l[i];
    T* orow = out + row[i];
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int d = 4 * (lane + 32 * n);
      if (d < D) Elem<T>::store(orow + d, acc[i][n].x * inv);
      if (d + 1 < D) Elem<T>::store(orow + d + 1, acc[i][n].y * inv);
      if (d + 2 < D) Elem<T>::store(orow + d + 2, acc[i][n].z * inv);
      if (d + 3 < D) Elem<T>::store(orow + d + 3, acc[i][n].w * inv);
    }
  }
}

struct Args {
  const void *q, *kv;
  void* out;
  const int *bt, *token_seq, *positions;
  int max_blocks, tokens, Hq, Hkv, D, page_size, window;
  float scale;
};
template <typename T, int NV, bool ASYNC, int WARPS, int BLOCKS>
int launch(const Args& a, cudaStream_t st) {
  static DeviceOnce once;
  if (!once.done()) {
    if (cudaFuncSetAttribute(paged_attention_generic_kernel<T, NV, ASYNC, WARPS, BLOCKS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             4 * smem_floats(NV == 1 ? 128 : MAX_D)) != cudaSuccess) {
      cudaGetLastError();
      return DIB_LAUNCH_FAILED;
    }
    once.mark();
  }
  const int group = a.Hq / a.Hkv;
  const long long blocks = ((long long)a.tokens * group + ITEMS - 1) / ITEMS;
  // 16 neighbouring queries touch at most this many tokens, and as many sequences
  int runs = (ITEMS + group - 2) / group + 1;
  if (runs > ITEMS) runs = ITEMS;
  if (runs > a.tokens) runs = a.tokens;
  dib_launch(paged_attention_generic_kernel<T, NV, ASYNC, WARPS, BLOCKS>, dim3((unsigned)(blocks * a.Hkv), runs), dim3(WARPS * 32),
             4 * smem_floats(a.D), st, (const T*)a.q, (T*)a.out, (const T*)a.kv, a.bt, a.max_blocks, a.token_seq, a.positions,
             a.tokens, a.Hq, a.Hkv, a.D, a.page_size, a.scale, a.window);
  DIB_CHECK_LAUNCH();
  return DIB_OK;
}

// Warps a block and blocks an SM, with the same bits.  The blocks that hold queries, some `busy` of them, come in waves of
// what the SMs hold; eight warps with all registers take the shortest time for one, fewer registers 1.04 of it, four
// warps of four queries 1.2, for groups of at most four heads (a decoding token's queries, one or two of the warps).  Heads
// above 128: one block an SM 1.0, two 1.08.  (us a layer, two / three blocks of eight warps / four of four: 64 sequences of 200 keys,
// 8 heads of 64 30 / 31 / 21, 128 of 300 82 / 68 / 55; 32 of 1,000, 12 heads of 96 133 / 80 / 87; a prompt of 1,000, bfloat16, 32 heads of
// 64 on one 570 / 493 / -.  Heads of 192, one / two blocks: 8 of 600, 16 heads 55 / 61, 32 of 1,000 337 / 196.)
template <typename T, bool ASYNC>
int choose(const Args& a, int decoded, cudaStream_t st) {
  const int group = a.Hq / a.Hkv, fit = 227 * 1024 / (4 * smem_floats(a.D) + 1024);
  const long long busy = ((long long)decoded + ((long long)(a.tokens - decoded) * group + ITEMS - 1) / ITEMS) * a.Hkv;
  auto time = [&](int blocks, float wave) {
    const long long at_once = 148ll * (blocks < fit ? blocks : fit);
    return (float)((busy + at_once - 1) / at_once) * wave;
  };
  if (a.D > 128) return time(2, 1.08f) < time(1, 1.f) ? launch<T, 2, ASYNC, 8, 2>(a, st) : launch<T, 2, ASYNC, 8, 1>(a, st);
  const float two = time(2, 1.f), three = time(3, 1.04f), four = group <= 4 && decoded == a.tokens ? time(4, 1.2f) : 1e30f;
  if (four < two && four < three) return launch<T, 1, ASYNC, 4, 4>(a, st);
  return three < two ? launch<T, 1, ASYNC, 8, 3>(a, st) : launch<T, 1, ASYNC, 8, 2>(a, st);
}

}  // namespace

// decoded: how many of the tokens are a sequence's only one in the step (for the choice of a form; any number is right)
extern "C" int dib_paged_attention_generic(const void* q, void* out, const void* kv_cache,
                                           const int* block_table, int max_blocks,
                                           const int* token_seq, const int* positions, int T, int decoded,
                                           int Hq, int Hkv, int D, int page_size, float scale,
                                           int window, int dtype, cudaStream_t st) {
  if (T == 0) return DIB_OK;
  if (D < 1 || D > MAX_D || Hkv < 1 || Hq % Hkv != 0 || page_size < 1) return DIB_BAD_SIZE;
  if (((long long)T * (Hq / Hkv) + ITEMS - 1) / ITEMS * Hkv > 0x7fffffffll) return DIB_BAD_SIZE;
  const Args a{q, kv_cache, out, block_table, token_seq, positions, max_blocks, T, Hq, Hkv, D, page_size, window, scale};
  decoded = decoded < 0 ? 0 : decoded > T ? T : decoded;
  if (dtype == 0)     // (rows of the cache start on 16 bytes when D is a multiple of 4)
    return D % 4 == 0 && ((uintptr_t)kv_cache & 15) == 0 ? choose<float, true>(a, decoded, st) : choose<float, false>(a, decoded, st);
  if (dtype == 1) return choose<__nv_bfloat16, false>(a, decoded, st);
  return DIB_BAD_DTYPE;
}

// The generalised delta rule of a prompt portion in chunks of 16 tokens, float32 throughout (heads of
// 64 or 128).  With G_i the product of the decays of a chunk's tokens up to i (per key channel) and S the
// state before the chunk, the recurrence
//   S_i = diag(w_i) S_(i-1) - b_i p_i + k_i v_i^T,   p_i = u_i^T S_(i-1),   o_i = S_i^T r_i
// unrolls to sums over the chunk's tokens:
//   p_i = (u_i G_(i-1))^T S + sum_(j<i) (K_ij v_j - A_ij p_j),
//   o_i = (r_i G_i)^T S + sum_(j<=i) (R_ij v_j - B_ij p_j),
//   S'  = diag(G) S + sum_j (G / G_j) (k_j v_j^T - b_j p_j),
// with A, B the products of u_i G_(i-1) and of r_i G_i with b_j / G_j, and K, R those with k_j / G_j.  The
// first two are solved for P = W S + P0 and O = Q S + O0 ahead of the states, for all chunks at once (forward
// substitution over 16 rows); what is left to do one chunk after the other are two products of 32 x D and
// D x 32 with a state's columns.  A chunk's log decay is 16 * decay_scale at most, so with |decay_scale| <=
// CHUNK_DECAY neither G nor 1 / G leaves float32's range, and every term of a sum is as exact as its factors.
#pragma once

#include <cuda_pipeline.h>

#include <type_traits>

#include "source.cuh"

namespace dchunks {

constexpr int CH = 16;                    // tokens of a chunk
constexpr float CHUNK_DECAY = 4.0f;       // e^(16 * 4) = 6e27
constexpr int COLS = 8;                   // value columns of a block that walks the chunks
constexpr int TP = 20;                    // row pitch of what is read 16 numbers of a row at a time
constexpr int RANKS = 64;                 // entries of the decay map's hidden vector at a time
// Tokens from which on a portion runs in chunks; shorter ones' token-by-token walk is over before the two kernels of
// this form have started up.  (From the projection to the output, us, token by token / chunks: 16 heads of 64, 64
// tokens 18.0 / 21.5, 256 tokens 40 / 33, 1,000 tokens 135 / 73, 2,048 tokens 275 / 145, 16 x 250 tokens 326 / 223;
// 8 heads of 128, 16 tokens 13.1 / 16.0, 64 tokens 23.6 / 19.5, 2,048 tokens 454 / 210, 16 x 250 tokens 384 / 322.)
constexpr int chunks_from(int D) { return D == 64 ? 112 : 48; }

// A chunk of a head in memory: W and Q ([32][D + 4]), G / G_j b_j (negated) and G / G_j k_j per channel
// ([D][TP] each), G [D]; then per group of 8 value columns P0, O0 ([16][8] each) and v ([8][TP]).
template <int D> struct Place {
  static constexpr int PITCH = D + 4;     // eight rows 16 bytes apart in the banks
  static constexpr int WQ = 2 * CH * PITCH;
  static constexpr int HEAD = WQ + 2 * D * TP + D;
  static constexpr int GROUP = 2 * CH * COLS + COLS * TP;
  static constexpr int FLOATS = HEAD + D / COLS * GROUP;
};

// Chunk c of sequence b has the place (cu[b] - cu[0]) / CH + b + c: no two share one, and no list is needed.
__device__ __forceinline__ int first_place(const int* cu, int b) { return (cu[b] - cu[0]) / CH + b; }
__device__ __forceinline__ bool chunk_at(const int* cu, int B, int place, int from, int& first, int& count) {
  int lo = 0, hi = B - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (first_place(cu, mid) <= place) lo = mid;
    else hi = mid - 1;
  }
  const int len = cu[lo + 1] - cu[lo], at = (place - first_place(cu, lo)) * CH;
  first = cu[lo] + at;
  count = min(CH, len - at);
  return count > 0 && len >= from;
}

// What a chunk needs of its tokens, from the projection to the solved sums: a block per (place, head), two
// threads a channel (eight tokens each) for the vectors, then one a column of W and one a column of P0.
// PROJ, W: as in delta_prepare_kernel, whose vectors these are (split sums: PROJ 2).
// Bound: by instructions (exponentials and divisions of the vectors, the decay map, the 16 rows one behind another) at a
// third of the issue rate, five blocks an SM: 54 us a layer of 2,048 tokens, 16 heads of 64, rank 64; with the map's
// rows and the hidden vectors asked for in turn 69 us.  The vectors alone, through memory, took 38.
template <int D, int PROJ, int W>
__global__ void __launch_bounds__(2 * D)
chunk_prepare_kernel(Source proj, const void* w2t, const float* w0, const float* a_bias, float* places,
                     const int* cu, int B, int from, int H, int R, float decay_scale, float key_eps) {
  constexpr int HALF = CH / 2, PITCH = Place<D>::PITCH, WARPS = D / 32;
  __shared__ __align__(16) float rows[4][CH][PITCH], vs[CH][PITCH];
  float (*ug)[PITCH] = rows[0], (*rg)[PITCH] = rows[1], (*bg)[PITCH] = rows[2], (*kg)[PITCH] = rows[3];
  __shared__ __align__(16) float pool[4 * CH * TP];
  // in their places until they are needed: a piece of w2t [RANKS][D], the hidden vectors' tanh [RANKS][16]
  static_assert(RANKS <= 4 * TP && RANKS * D <= 4 * CH * PITCH, "the pieces fit");
  using WT = typename std::conditional<W == 1, __nv_bfloat16, float>::type;
  WT (*wt)[D] = reinterpret_cast<WT (*)[D]>(&rows[0][0][0]);
  float (*th)[CH] = reinterpret_cast<float (*)[CH]>(pool);
  float (*mat)[CH][TP] = reinterpret_cast<float (*)[CH][TP]>(pool);      // A, K, B, R
  __shared__ float sums[CH][WARPS], g_mid[D], g_all[D];
  pdl_trigger();
  const int h = blockIdx.y, c = threadIdx.x % D, half = threadIdx.x / D, i0 = half * HALF;
  const int HD = H * D, ch = h * D + c;
  const long long width = 5 * HD + R;
  auto fetch_map = [&](int j0) {       // rows j0 .. of the decay map, this head's channels (16 bytes a copy)
    constexpr int E = 16 / sizeof(WT), PER = D / E;
    const int n = min(RANKS, R - j0);
    for (int e = threadIdx.x; e < n * PER; e += 2 * D)
      __pipeline_memcpy_async(&wt[e / PER][e % PER * E],
                              reinterpret_cast<const WT*>(w2t) + (long long)(j0 + e / PER) * HD + h * D + e % PER * E, 16);
    __pipeline_commit();
  };
  fetch_map(0);                        // (a constant: ahead of the wait)
  pdl_wait(proj.p);
  int first, count;
  if (!chunk_at(cu, B, blockIdx.x, from, first, count)) return;
  auto element = [&](long long at) {
    if constexpr (PROJ == 0) return reinterpret_cast<const float*>(proj.p)[at];
    else if constexpr (PROJ == 1) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(proj.p)[at]);
    else return source_load(proj, at);
  };
  float r[HALF], k[HALF], a[HALF], z[HALF];
  {
    float v[HALF];
#pragma unroll
    for (int i = 0; i < HALF; ++i) {
      const bool in = i0 + i < count;
      const long long row = (first + i0 + i) * width + ch;
      r[i] = in ? element(row) : 0.f;
      k[i] = in ? element(row + HD) : 0.f;
      v[i] = in ? element(row + 2 * HD) : 0.f;
      a[i] = in ? element(row + 4 * HD) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < HALF; ++i) vs[i0 + i][c] = v[i];
  }
  float hid[RANKS * CH / (2 * D)];     // the first piece's hidden vectors
  auto hidden = [&](int j0, int q) {
    const int e = threadIdx.x + q * 2 * D, i = e / RANKS, j = e % RANKS;
    return i < count && j0 + j < R ? element((first + i) * width + 5 * HD + j0 + j) : 0.f;
  };
#pragma unroll
  for (int q = 0; q < RANKS * CH / (2 * D); ++q) hid[q] = hidden(0, q);
#pragma unroll
  for (int i = 0; i < HALF; ++i) {
    z[i] = 0.f;
    const float part = warp_sum(k[i] * k[i]);
    if ((c & 31) == 0) sums[i0 + i][c >> 5] = part;
  }
  for (int j0 = 0; j0 < R; j0 += RANKS) {
    const int n = min(RANKS, R - j0);
    if (j0 > 0) {
      __syncthreads();
      fetch_map(j0);
    }
#pragma unroll
    for (int q = 0; q < RANKS * CH / (2 * D); ++q) {
      const int e = threadIdx.x + q * 2 * D;
      th[e % RANKS][e / RANKS] = tanhf(j0 > 0 ? hidden(j0, q) : hid[q]);
    }
    __pipeline_wait_prior(0);
    __syncthreads();
#pragma unroll 8
    for (int j = 0; j < n; ++j) {
      const float w = load_as(wt, W, j * D + c);
      const float4 x = *reinterpret_cast<const float4*>(&th[j][i0]), y = *reinterpret_cast<const float4*>(&th[j][i0 + 4]);
      z[0] = __fmaf_rn(w, x.x, z[0]);
      z[1] = __fmaf_rn(w, x.y, z[1]);
      z[2] = __fmaf_rn(w, x.z, z[2]);
      z[3] = __fmaf_rn(w, x.w, z[3]);
      z[4] = __fmaf_rn(w, y.x, z[4]);
      z[5] = __fmaf_rn(w, y.y, z[5]);
      z[6] = __fmaf_rn(w, y.z, z[6]);
      z[7] = __fmaf_rn(w, y.w, z[7]);
    }
  }
  // decays (1 behind the sequence's last token, where every other vector is 0) and their products
  const float bias_w = w0[ch], bias_a = a_bias != nullptr ? a_bias[ch] : 0.f;
  float g = 1.f;
#pragma unroll
  for (int i = 0; i < HALF; ++i) {
    if (i0 + i < count) g *= expf(-decay_scale * sigmoid_f32(__fadd_rn(z[i], bias_w)));
    z[i] = g;
  }
  if (half == 0) g_mid[c] = g;
  __syncthreads();
  float before = 1.f;                                            // G_(i-1)
  if (half == 1) {
    before = g_mid[c];
    g_all[c] = before * g;
  }
  float* place = places + ((long long)blockIdx.x * H + h) * Place<D>::FLOATS;
#pragma unroll
  for (int i = 0; i < HALF; ++i) {
    float ss = 0.f;
#pragma unroll
    for (int x = 0; x < WARPS; ++x) ss += sums[i0 + i][x];
    const float now = half == 1 ? g_mid[c] * z[i] : z[i], inv = 1.0f / now;
    const bool in = i0 + i < count;
    const float u = k[i] / sqrtf(ss + key_eps);
    const float b = in ? sigmoid_f32(__fadd_rn(a[i], bias_a)) * u : 0.f;
    ug[i0 + i][c] = in ? u * before : 0.f;
    rg[i0 + i][c] = r[i] * now;
    bg[i0 + i][c] = a[i] = b * inv;
    kg[i0 + i][c] = k[i] = k[i] * inv;
    before = now;
  }
  __syncthreads();
  {
    const float all = g_all[c];
    if (half == 0) place[Place<D>::WQ + 2 * D * TP + c] = all;
    float4* to = reinterpret_cast<float4*>(place + Place<D>::WQ + c * TP + i0);
    to[0] = make_float4(-(a[0] * all), -(a[1] * all), -(a[2] * all), -(a[3] * all));
    to[1] = make_float4(-(a[4] * all), -(a[5] * all), -(a[6] * all), -(a[7] * all));
    to += D * TP / 4;
    to[0] = make_float4(k[0] * all, k[1] * all, k[2] * all, k[3] * all);
    to[1] = make_float4(k[4] * all, k[5] * all, k[6] * all, k[7] * all);
  }
  // [u G ; r G] times [b / G ; k / G]: a thread takes rows i of both and columns j, j + 8 of both; the
  // threads beyond 128 (heads of 128) the second half of the channels
  {
    constexpr int PARTS = D / 64;
    const int t = threadIdx.x & 127, part = threadIdx.x >> 7, i = t >> 3, j = t & 7;
    float2 acc[2][4] = {};
#pragma unroll 4
    for (int d = part * 64; d < part * 64 + 64; d += 4) {
      const float4 x[2] = {*reinterpret_cast<const float4*>(&ug[i][d]), *reinterpret_cast<const float4*>(&rg[i][d])};
      const float4 y[4] = {*reinterpret_cast<const float4*>(&bg[j][d]), *reinterpret_cast<const float4*>(&bg[j + 8][d]),
                           *reinterpret_cast<const float4*>(&kg[j][d]), *reinterpret_cast<const float4*>(&kg[j + 8][d])};
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          acc[m][n] = __ffma2_rn(make_float2(x[m].x, x[m].y), make_float2(y[n].x, y[n].y), acc[m][n]);
          acc[m][n] = __ffma2_rn(make_float2(x[m].z, x[m].w), make_float2(y[n].z, y[n].w), acc[m][n]);
        }
    }
#pragma unroll
    for (int p = PARTS - 1; p >= 0; --p) {
      if (p == part) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int n = 0; n < 4; ++n) {
            const int jj = j + (n & 1) * 8;
            float* at = &mat[m * 2 + (n >> 1)][i][jj];
            float s = __fadd_rn(acc[m][n].x, acc[m][n].y);
            if (p < PARTS - 1) s = __fadd_rn(s, *at);
            *at = (m == 0 ? jj < i : jj <= i) ? s : 0.f;
          }
      }
      __syncthreads();
    }
  }
  // rows in turn, in registers: x_i = known_i - sum_(j<i) A_ij x_j (W with known = u G, P0 with known = K v)
  float2 x[HALF], v[HALF];
  const bool second = half == 1;
#pragma unroll
  for (int i = 0; i < HALF; ++i) {
    x[i] = make_float2(0.f, 0.f);
    v[i] = second ? make_float2(vs[2 * i][c], vs[2 * i + 1][c]) : make_float2(0.f, 0.f);
  }
  // sum over j < n of m_j y_j, even and odd j apart (nothing behind n is touched: a token does not see later ones)
  auto dot = [](const float* m, const float2 (&y)[HALF], int n, float2 s) {
#pragma unroll
    for (int q = 0; q < CH / 4; ++q) {
      if (4 * q >= n) break;
      const float4 f = *reinterpret_cast<const float4*>(m + 4 * q);
      if (4 * q + 1 < n) s = __ffma2_rn(make_float2(f.x, f.y), y[2 * q], s);
      else s.x = __fmaf_rn(f.x, y[2 * q].x, s.x);
      if (4 * q + 3 < n) s = __ffma2_rn(make_float2(f.z, f.w), y[2 * q + 1], s);
      else if (4 * q + 2 < n) s.x = __fmaf_rn(f.z, y[2 * q + 1].x, s.x);
    }
    return s;
  };
  const float2 zero = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    const float2 minus = dot(mat[0][i], x, i, zero);
    float known;
    if (second) {
      const float2 plus = dot(mat[1][i], v, i, zero);
      known = __fadd_rn(plus.x, plus.y);
    } else {
      known = ug[i][c];
    }
    const float xi = __fsub_rn(known, __fadd_rn(minus.x, minus.y));
    if (i & 1) x[i >> 1].y = xi;
    else x[i >> 1].x = xi;
  }
  float* group = place + Place<D>::HEAD + (c / COLS) * Place<D>::GROUP;
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    const float2 minus = dot(mat[2][i], x, i + 1, zero);
    float known;
    if (second) {
      const float2 plus = dot(mat[3][i], v, i + 1, zero);
      known = __fadd_rn(plus.x, plus.y);
    } else {
      known = rg[i][c];
    }
    const float xi = i & 1 ? x[i >> 1].y : x[i >> 1].x;
    const float yi = __fsub_rn(known, __fadd_rn(minus.x, minus.y));
    if (second) {
      group[i * COLS + c % COLS] = xi;
      group[(CH + i) * COLS + c % COLS] = yi;
    } else {
      place[i * PITCH + c] = xi;
      place[(CH + i) * PITCH + c] = yi;
    }
  }
  if (second) {
    float4* to = reinterpret_cast<float4*>(group + 2 * CH * COLS + c % COLS * TP);
#pragma unroll
    for (int q = 0; q < CH / 4; ++q) to[q] = make_float4(v[2 * q].x, v[2 * q].y, v[2 * q + 1].x, v[2 * q + 1].y);
  }
}

// The chunks of a sequence one after the other: a block per (sequence, head, 8 CPT value columns), a warp per 16
// state rows; a thread keeps rows 16 warp + lane / 8 + 4 r (r < 4) of columns lane % 8 + 8 u (u < CPT).  Per chunk:
// every warp's share of W S and Q S over its own rows (its states through shared memory, nobody else's), the warps'
// shares added in warp order together with P0 and O0, then the states.  One more warp brings the chunks into shared
// memory, two ahead of the one that is worked on.  CPT: with one column a thread more blocks share a sequence's
// work; with two every block's copies serve twice the columns, for steps that fill the GPU either way.  A column's
// sums are the same.  Bound: by latency, a chunk's two products with two barriers behind one another, 0.6 us
// (2,048 tokens, 16 heads of 64: 80 us; token by token 229; copies by the warps that compute 100; a warp per 8 state rows 90).
constexpr int STAGES = 4;
template <int D, int CPT> constexpr size_t walk_smem() {
  return sizeof(float) * (STAGES * (Place<D>::HEAD + CPT * Place<D>::GROUP) +
                          CPT * (D / 16 * (2 * CH * COLS + COLS * TP) + COLS * TP));
}
template <int D, int CPT>
__global__ void __launch_bounds__(2 * D + 32, 2)
chunk_walk_kernel(const float* places, float* state, long long slot_stride, float* o_out, const int* cu,
                  const int* state_slots, int from_tokens, int H) {
  using P = Place<D>;
  constexpr int THREADS = 2 * D, WARPS = D / 16, STAGE = P::HEAD + CPT * P::GROUP, NC = COLS * CPT;
  extern __shared__ __align__(16) float walk_smem_[];
  float* red = walk_smem_ + STAGES * STAGE;                      // [WARPS][32][NC]: the warps' shares
  float* own = red + WARPS * 2 * CH * NC;                        // [WARPS][NC][TP]: a warp's states
  float* pt = own + WARPS * NC * TP;                             // [NC][TP]: the chunk's p, by column
  const int b = blockIdx.x, h = blockIdx.y, group = blockIdx.z * CPT;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_wait(places);                  // (launched in stream order)
  const int t0 = cu[b], t1 = cu[b + 1];
  if (t1 <= t0 || t1 - t0 < from_tokens) return;
  const int chunks = (t1 - t0 + CH - 1) / CH;
  if (warp == WARPS) {               // the copies
    const long long step = (long long)H * P::FLOATS;
    const float* from = places + ((long long)first_place(cu, b) * H + h) * P::FLOATS + 4 * lane;
    auto fetch = [&](int n) {
      if (n < chunks) {
        float* to = walk_smem_ + n % STAGES * STAGE + 4 * lane;
        const float* src = from + n * step;
#pragma unroll 8
        for (int i = 0; i < P::HEAD / 128; ++i) __pipeline_memcpy_async(to + 128 * i, src + 128 * i, 16);
        if (4 * lane < P::HEAD % 128) __pipeline_memcpy_async(to + P::HEAD / 128 * 128, src + P::HEAD / 128 * 128, 16);
        to += P::HEAD;
        src += P::HEAD + group * P::GROUP;
#pragma unroll
        for (int i = 0; 128 * i < CPT * P::GROUP; ++i)
          if (128 * i + 4 * lane < CPT * P::GROUP) __pipeline_memcpy_async(to + 128 * i, src + 128 * i, 16);
      }
      __pipeline_commit();           // (an empty group past the end keeps the count)
    };
    fetch(0);
    fetch(1);
    fetch(2);
    __pipeline_wait_prior(2);
    __syncthreads();                 // chunk 0 has landed
    for (int n = 0; n < chunks; ++n) {
      __pipeline_wait_prior(1);
      __syncthreads();               // chunk n + 1 has landed; everybody is done with chunk n - 1
      fetch(n + 3);                  // into its place
    }
    __pipeline_wait_prior(0);
    return;
  }
  const long long slot = state_slots[b];
  const bool kept = slot != 0;       // slot 0 belongs to padding sequences: zero state, nothing stored
  const int row = warp * 16 + (lane >> 3), col = lane & 7;
  float* S = state + slot * slot_stride + ((long long)h * D + row) * D + group * COLS + col;
  float st[CPT][4];
  float* mine = own + warp * NC * TP;
  auto share = [&] {
#pragma unroll
    for (int u = 0; u < CPT; ++u)
#pragma unroll
      for (int r = 0; r < 4; ++r) mine[(col + COLS * u) * TP + (lane >> 3) + 4 * r] = st[u][r];
    __syncwarp();
  };
#pragma unroll
  for (int u = 0; u < CPT; ++u)
#pragma unroll
    for (int r = 0; r < 4; ++r) st[u][r] = kept ? S[4 * r * D + COLS * u] : 0.f;
  share();
  __syncthreads();
  const int pi = lane >> 2, pc = 2 * (lane & 3);       // a thread's rows pi + 8 r, columns pc + 8 u and the next
  float* o_at = o_out + ((long long)t0 * H + h) * D + group * COLS;
  for (int n = 0; n < chunks; ++n) {
    const float* at = walk_smem_ + n % STAGES * STAGE;
    const float* mid = at + P::HEAD;
    float2 acc[CPT][4][2] = {};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float4 w[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) w[r] = *reinterpret_cast<const float4*>(at + (pi + 8 * r) * P::PITCH + warp * 16 + 4 * q);
#pragma unroll
      for (int u = 0; u < CPT; ++u)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float4 s = *reinterpret_cast<const float4*>(mine + (pc + e + COLS * u) * TP + 4 * q);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            acc[u][r][e] = __ffma2_rn(make_float2(w[r].x, w[r].y), make_float2(s.x, s.y), acc[u][r][e]);
            acc[u][r][e] = __ffma2_rn(make_float2(w[r].z, w[r].w), make_float2(s.z, s.w), acc[u][r][e]);
          }
        }
    }
#pragma unroll
    for (int u = 0; u < CPT; ++u)
#pragma unroll
      for (int r = 0; r < 4; ++r)
        *reinterpret_cast<float2*>(red + (warp * 2 * CH + pi + 8 * r) * NC + pc + COLS * u) =
            make_float2(__fadd_rn(acc[u][r][0].x, acc[u][r][0].y), __fadd_rn(acc[u][r][1].x, acc[u][r][1].y));
    asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");       // the warps' shares are there
#pragma unroll
    for (int e0 = 0; e0 < 2 * CH * NC; e0 += THREADS) {
      const int e = e0 + tid, i = e / NC, cc = e % NC;
      float s = red[e];
#pragma unroll
      for (int w = 1; w < WARPS; ++w) s = __fadd_rn(s, red[w * 2 * CH * NC + e]);
      s = __fadd_rn(s, mid[cc / COLS * P::GROUP + i * COLS + cc % COLS]);
      if (i < CH) pt[cc * TP + i] = s;
      else if (n * CH + i - CH < t1 - t0) o_at[(long long)(n * CH + i - CH) * H * D + cc] = s;
    }
    __syncthreads();                 // p is there, and the next chunk
    float2 sum[CPT][4] = {};
    const float* bk = at + P::WQ + row * TP;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float4 p[CPT], v[CPT];
#pragma unroll
      for (int u = 0; u < CPT; ++u) {
        p[u] = *reinterpret_cast<const float4*>(pt + (col + COLS * u) * TP + 4 * q);
        v[u] = *reinterpret_cast<const float4*>(mid + u * P::GROUP + 2 * CH * COLS + col * TP + 4 * q);
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float4 x = *reinterpret_cast<const float4*>(bk + 4 * r * TP + 4 * q);
        const float4 y = *reinterpret_cast<const float4*>(bk + (D + 4 * r) * TP + 4 * q);
#pragma unroll
        for (int u = 0; u < CPT; ++u) {
          sum[u][r] = __ffma2_rn(make_float2(x.x, x.y), make_float2(p[u].x, p[u].y), sum[u][r]);
          sum[u][r] = __ffma2_rn(make_float2(y.x, y.y), make_float2(v[u].x, v[u].y), sum[u][r]);
          sum[u][r] = __ffma2_rn(make_float2(x.z, x.w), make_float2(p[u].z, p[u].w), sum[u][r]);
          sum[u][r] = __ffma2_rn(make_float2(y.z, y.w), make_float2(v[u].z, v[u].w), sum[u][r]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float g = at[P::WQ + 2 * D * TP + row + 4 * r];
#pragma unroll
      for (int u = 0; u < CPT; ++u) st[u][r] = __fmaf_rn(g, st[u][r], __fadd_rn(sum[u][r].x, sum[u][r].y));
    }
    share();
  }
#pragma unroll
  for (int u = 0; u < CPT; ++u)
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (kept) S[4 * r * D + COLS * u] = st[u][r];
}

}  // namespace dchunks

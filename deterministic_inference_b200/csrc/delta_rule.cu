// Generalised delta rule with a decay per key channel: per head a state S [D keys, D values]
// in float32, carried from token to token in the request's state slot,
//   S_t = diag(w_t) S_(t-1) - (a_t * u_t) (u_t^T S_(t-1)) + k_t v_t^T,   o_t = S_t^T r_t,
// with u = k / sqrt(sum(k^2) + key_eps) the unit key, w = exp(-decay_scale * sigmoid(lora + w0))
// the decay and a = sigmoid(. + bias) the removal rate.  Three kernels: the per-token vectors
// (all float32), the recurrence, and the output (per-head RMS norm, weight, sigmoid gate).
//
// The recurrence kernels take a state of D key rows by E value columns per head and a token's
// vectors as [w | b | u | k | r] of D elements each and v of E:
//   S_t = diag(w) S_(t-1) - b (u^T S_(t-1)) + k v^T,   o_t = S_t^T r,
// which is also the gated delta rule (S <- g S; S <- S + beta k (v - S^T k)^T) with w = g in
// every row, u = the unit key, b = g beta u and k = beta u.  Its per-token vectors (short causal
// convolutions with silu in front of q, k and v, unit vectors, rate and decay) and its output
// (RMS norm over a head, weight, silu gate) have kernels of their own below.
#include <cuda_pipeline.h>

#include <type_traits>

#include "source.cuh"
#include "conv_tail.cuh"

// proj row: [r | k | v | g | a_pre | lora hidden] = 5 * H * D + R columns; w2t [R][H * D] (the
// decay map's second matrix, transposed: the threads of a block read consecutive elements).
// packed [T][H][6][D] float32: w, a * u, u, k, r, v.
// A block takes TOKENS tokens of a head: an element of w2t is read once for all of them, and all their
// projected elements are asked for before the first is used, of split sums (PROJ 2) a split of all of
// them at a time.  PROJ 0 / 1: proj is a stored float32 / bfloat16 matrix; W: w2t's type.  A token's
// vectors are the same in every form, which the launcher picks by what is quickest.  Bound: by latency
// below some hundred tokens (the chain over R), then by the 48 bytes written for a channel and token.
// (16 heads of 64, R = 64, us: split sums, one token a block, 1 / 8 / 64 tokens of eight splits 4.0 / 4.2 / 8.2;
// eight tokens a block and the splits an element at a time 10.3 / 51 / 47.  Stored, two / four tokens a
// block: 8 tokens 3.9 / 5.7, 128 tokens 7.4 / 9.9, 256 tokens 8.3 / 10.3, 512 tokens 13.3 / 11.8, 2,048
// tokens 46 / 34; eight 10.2, 11.2, 14.9, 16, 38.)
constexpr int PREP_RANKS = 512;                       // entries of the hidden vector at a time
constexpr int PREP_FOUR_FROM = 384;                   // tokens from which on a block takes four
// (The second bound of the launch leaves the compiler the registers that sixteen weights in flight need.)
template <int TOKENS, int PROJ, int W>
__global__ void __launch_bounds__(TOKENS == 1 ? 1024 : 256, TOKENS == 1 ? 1 : 4)
delta_prepare_kernel(Source proj, const void* w2t, const float* w0, const float* a_bias, float* packed, int T, int H,
                     int D, int R, float decay_scale, float key_eps) {
  __shared__ __align__(16) float th[PREP_RANKS * TOKENS];            // tanh of the lora hidden
  __shared__ float sums[TOKENS * 32];                                // the warps' sums of squares
  pdl_prologue();
  const int t0 = blockIdx.x * TOKENS, h = blockIdx.y, c = threadIdx.x;
  const int tokens = min(TOKENS, T - t0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int HD = H * D;
  const long long width = 5 * HD + R;
  auto element = [&](long long at) {
    if constexpr (PROJ == 0) return reinterpret_cast<const float*>(proj.p)[at];
    else if constexpr (PROJ == 1) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(proj.p)[at]);
    else return source_load(proj, at);
  };
  const int ch = h * D + c;
  float r[TOKENS], k[TOKENS], v[TOKENS], a[TOKENS], z[TOKENS];
  if constexpr (PROJ == 2) {
    static_assert(TOKENS == 1, "split sums are a few tokens'");
    r[0] = k[0] = v[0] = a[0] = -0.f;                  // (-0 plus the first split is that split)
    if (c < D) {
      const float* f = reinterpret_cast<const float*>(proj.p) + t0 * width + ch;
#pragma unroll 4
      for (int sp = 0; sp < proj.splits; ++sp, f += proj.stride) {
        r[0] = __fadd_rn(r[0], f[0]);
        k[0] = __fadd_rn(k[0], f[HD]);
        v[0] = __fadd_rn(v[0], f[2 * HD]);
        a[0] = __fadd_rn(a[0], f[4 * HD]);
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < TOKENS; ++i) {
      const bool in = c < D && i < tokens;
      const long long row = (t0 + i) * width + ch;
      r[i] = in ? element(row) : 0.f;
      k[i] = in ? element(row + HD) : 0.f;
      v[i] = in ? element(row + 2 * HD) : 0.f;
      a[i] = in ? element(row + 4 * HD) : 0.f;
    }
  }
#pragma unroll
  for (int i = 0; i < TOKENS; ++i) {
    z[i] = 0.f;
    const float part = warp_sum(k[i] * k[i]);
    if (lane == 0) sums[i * 32 + warp] = part;
  }
  for (int j0 = 0; j0 < R; j0 += PREP_RANKS) {
    const int n = min(PREP_RANKS, R - j0);
    if (j0 > 0) __syncthreads();
    for (int e = threadIdx.x; e < n * TOKENS; e += blockDim.x) {
      const int i = e / n, j = e - i * n;
      th[j * TOKENS + i] = i < tokens ? tanhf(element((t0 + i) * width + 5 * HD + j0 + j)) : 0.f;
    }
    __syncthreads();
    if (c < D) {
#pragma unroll 16
      for (int j = 0; j < n; ++j) {
        const float w = load_as(w2t, W, (long long)(j0 + j) * HD + ch);
        if constexpr (TOKENS == 1) {
          z[0] = __fmaf_rn(w, th[j], z[0]);
        } else if constexpr (TOKENS == 2) {
          const float2 y = *reinterpret_cast<const float2*>(th + j * 2);
          z[0] = __fmaf_rn(w, y.x, z[0]);
          z[1] = __fmaf_rn(w, y.y, z[1]);
        } else {
          const float4 y = *reinterpret_cast<const float4*>(th + j * 4);
          z[0] = __fmaf_rn(w, y.x, z[0]);
          z[1] = __fmaf_rn(w, y.y, z[1]);
          z[2] = __fmaf_rn(w, y.z, z[2]);
          z[3] = __fmaf_rn(w, y.w, z[3]);
        }
      }
    }
  }
  __syncthreads();                 // (R may be 0)
  if (c >= D) return;
  const float bias_w = w0[ch], bias_a = a_bias != nullptr ? a_bias[ch] : 0.f;
#pragma unroll
  for (int i = 0; i < TOKENS; ++i) {
    if (i >= tokens) break;
    float ss = 0.f;
    for (int x = 0; x < warps; ++x) ss += sums[i * 32 + x];
    const float rate = sigmoid_f32(__fadd_rn(a[i], bias_a));
    const float u = k[i] / sqrtf(ss + key_eps);
    float* out = packed + ((long long)(t0 + i) * H + h) * 6 * D + c;
    out[0] = expf(-decay_scale * sigmoid_f32(__fadd_rn(z[i], bias_w)));
    out[D] = rate * u;
    out[2 * D] = u;
    out[3 * D] = k[i];
    out[4 * D] = r[i];
    out[5 * D] = v[i];
  }
}

// One warp per (sequence, head, 8 value columns); a column's D state rows are spread over
// 4 lanes (row i = 16 q + 4 s + e for lane s), each lane keeping its rows in registers over
// all tokens of the sequence in this step.  Each of the two sums over the rows (u . S and
// r . S) is taken as four chains inside a lane (rows e, e + 16, e + 32, ... for e = 0..3, in
// ascending order), added as (c0 + c1) + (c2 + c3), and then over the 4 lanes by a butterfly:
// an order that depends on D alone.  Every warp stages the token's six vectors in a ring of
// its own in shared memory by asynchronous copies, DR_STAGES tokens deep, and waits for nobody
// but itself.
template <int MAXR, int DR_STAGES>
__global__ void __launch_bounds__(128)
delta_recurrence_kernel(const float* packed, float* state, long long slot_stride, float* o_out,
                        const int* cu_q_lens, const int* state_slots, int H, int D, int E) {
  extern __shared__ __align__(16) float dr_smem[];           // [4 warps][DR_STAGES][5 Dp + Ep]
  const int Dp = (D + 15) / 16 * 16, Ep = (E + 15) / 16 * 16;
  const int SV = 5 * Dp + Ep;                  // a stage: w, b, u, k, r of Dp floats each, then v of Ep
  const int NR = Dp / 4;                       // rows per lane (<= MAXR)
  const int b = blockIdx.x, h = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int s = lane & 3;
  const int c = (blockIdx.z * 4 + warp) * 8 + (lane >> 2);
  const bool active = c < E;
  if ((blockIdx.z * 4 + warp) * 8 >= E) return;              // none of this warp's columns exists
  float* ring = dr_smem + warp * DR_STAGES * SV;
  if (Dp != D)
    for (int i = lane; i < DR_STAGES * SV; i += 32) ring[i] = 0.f;   // the padding stays 0
  pdl_wait();                        // (the kernel behind this one is not launched ahead of its end)
  const int t0 = cu_q_lens[b], t1 = cu_q_lens[b + 1];
  if (t1 <= t0) return;
  const long long slot = state_slots[b];
  const bool kept = slot != 0;       // slot 0 belongs to padding sequences: zero state, nothing stored
  float* S = state + slot * slot_stride + (long long)h * D * E;
  float st[MAXR];
#pragma unroll
  for (int ii = 0; ii < MAXR; ++ii) {
    const int i = (ii >> 2) * 16 + s * 4 + (ii & 3);
    st[ii] = (kept && ii < NR && active && i < D) ? S[(long long)i * E + c] : 0.f;
  }
  __syncwarp();
  const int PV = 5 * D + E;                    // a token's vectors of one head, as they are stored
  const bool wide = ((D | E) & 3) == 0;        // every vector starts on 16 bytes
  // this lane's 16-byte pieces of a token's vectors: where they come from and go to
  constexpr int PIECES = MAXR * 4 * 6 / 4 / 32;      // (5 D + E) / 4 pieces over 32 lanes, at most
  int src_at[PIECES], dst_at[PIECES];
#pragma unroll
  for (int k = 0; k < PIECES; ++k) {
    const int at = (lane + 32 * k) * 4;
    const int vsel = at < 5 * D ? at / D : 5, d = at - vsel * D;
    src_at[k] = (wide && at < PV) ? at : -1;
    dst_at[k] = vsel * Dp + d;
  }
  auto prefetch = [&](int t, int stage) {
    if (t < t1) {
      const float* src = packed + ((long long)t * H + h) * PV;
      float* dst = ring + stage * SV;
      if (wide) {
#pragma unroll
        for (int k = 0; k < PIECES; ++k)
          if (src_at[k] >= 0) __pipeline_memcpy_async(dst + dst_at[k], src + src_at[k], 16);
      } else {
        for (int i = lane; i < PV; i += 32) {
          const int vsel = i < 5 * D ? i / D : 5, d = i - vsel * D;
          __pipeline_memcpy_async(dst + vsel * Dp + d, src + i, 4);
        }
      }
    }
    __pipeline_commit();                       // (an empty group past the end keeps the count)
  };
#pragma unroll
  for (int k = 0; k < DR_STAGES - 1; ++k) prefetch(t0 + k, k);
  for (int t = t0; t < t1; ++t) {
    const int stage = (t - t0) % DR_STAGES;
    prefetch(t + DR_STAGES - 1, (stage + DR_STAGES - 1) % DR_STAGES);
    __pipeline_wait_prior(DR_STAGES - 1);
    __syncwarp();
    const float* vw = ring + stage * SV;
    const float* vb = vw + Dp;
    const float* vu = vb + Dp;
    const float* vk = vu + Dp;
    const float* vr = vk + Dp;
    const float v = active ? vr[Dp + c] : 0.f;
    float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
#pragma unroll
    for (int q = 0; q < MAXR / 4; ++q) {
      if (q * 4 < NR) {
        const float4 u4 = *reinterpret_cast<const float4*>(vu + q * 16 + s * 4);
        d0 = __fmaf_rn(u4.x, st[q * 4 + 0], d0);
        d1 = __fmaf_rn(u4.y, st[q * 4 + 1], d1);
        d2 = __fmaf_rn(u4.z, st[q * 4 + 2], d2);
        d3 = __fmaf_rn(u4.w, st[q * 4 + 3], d3);
      }
    }
    float dot = __fadd_rn(__fadd_rn(d0, d1), __fadd_rn(d2, d3));
    dot = __fadd_rn(dot, __shfl_xor_sync(0xffffffffu, dot, 1));
    dot = __fadd_rn(dot, __shfl_xor_sync(0xffffffffu, dot, 2));
    float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
    for (int q = 0; q < MAXR / 4; ++q) {
      if (q * 4 < NR) {
        const int at = q * 16 + s * 4;
        const float4 w4 = *reinterpret_cast<const float4*>(vw + at);
        const float4 b4 = *reinterpret_cast<const float4*>(vb + at);
        const float4 k4 = *reinterpret_cast<const float4*>(vk + at);
        const float4 r4 = *reinterpret_cast<const float4*>(vr + at);
        float n0 = __fmaf_rn(k4.x, v, __fmaf_rn(-b4.x, dot, __fmul_rn(w4.x, st[q * 4 + 0])));
        float n1 = __fmaf_rn(k4.y, v, __fmaf_rn(-b4.y, dot, __fmul_rn(w4.y, st[q * 4 + 1])));
        float n2 = __fmaf_rn(k4.z, v, __fmaf_rn(-b4.z, dot, __fmul_rn(w4.z, st[q * 4 + 2])));
        float n3 = __fmaf_rn(k4.w, v, __fmaf_rn(-b4.w, dot, __fmul_rn(w4.w, st[q * 4 + 3])));
        st[q * 4 + 0] = n0; st[q * 4 + 1] = n1; st[q * 4 + 2] = n2; st[q * 4 + 3] = n3;
        o0 = __fmaf_rn(r4.x, n0, o0);
        o1 = __fmaf_rn(r4.y, n1, o1);
        o2 = __fmaf_rn(r4.z, n2, o2);
        o3 = __fmaf_rn(r4.w, n3, o3);
      }
    }
    float o = __fadd_rn(__fadd_rn(o0, o1), __fadd_rn(o2, o3));
    o = __fadd_rn(o, __shfl_xor_sync(0xffffffffu, o, 1));
    o = __fadd_rn(o, __shfl_xor_sync(0xffffffffu, o, 2));
    if (active && s == 0) o_out[((long long)t * H + h) * E + c] = o;
    __syncwarp();        // the next round's copies overwrite the stage that was read one round ago
  }
#pragma unroll
  for (int ii = 0; ii < MAXR; ++ii) {
    const int i = (ii >> 2) * 16 + s * 4 + (ii & 3);
    if (kept && ii < NR && active && i < D) S[(long long)i * E + c] = st[ii];
  }
}

// The same recurrence with a column's rows over LANES = 16 lanes (row i = 64 q + 4 s + e for lane s),
// CPT columns a thread, WARPS warps a block per (sequence, head, 32 / LANES * CPT * WARPS value
// columns).  The form for steps with few sequences and many tokens (prompt portions): few warps a
// scheduler, so a token takes what its instructions and the chain from its state to the next one's
// take (the row sum's FMA, four exchanges between lanes, one FMA).  Nothing else stands in that
// chain: a token's vectors are in registers before, w S + k v is ready when the sum arrives, and the output's exchanges run one token
// behind, side by side with the sum's.  One more warp brings the vectors into shared memory,
// DR_TOKENS tokens at a time, one group ahead, with one barrier a group; strides are constants of
// the instance (D and E padded with zeros to LANES * MAXR).  Its sums are ordered differently from
// the form above (four chains by e, then a butterfly over 16 lanes), again by D alone.
// NEXT: the next token's vectors are read while one is worked on; not with D or E above 128, where two
// tokens' take all registers there are and half as many warps fit an SM (4 heads of 256, 8 x 64 tokens:
// 140 us, read in their turn 103; 16 heads of 200, 16 x 64 tokens: 783 and 554; one sequence of 256
// tokens, 4 heads of 256: 132 and 125).
// (2,048 tokens, 16 heads of 64: 230 us, rows over 8 lanes 344, over 4 649 us; 8 heads of 128: 412 us;
// 4 heads of 256: 968 us.  Copies by the warps that compute, a barrier a token and both exchanges in the
// chain: 864, 907 and 1,102 us; 16 x 64 tokens, 16 heads of 200: 646 us.)
template <int Q, int CPT> struct DeltaToken {      // a lane's part of a token's vectors
  float4 w[Q], b[Q], u[Q], k[Q], r[Q];
  float v[CPT];
};
template <int MAXR, int LANES, int CPT, int WARPS, int DR_TOKENS, int DR_STAGES, bool NEXT>
__global__ void __launch_bounds__(32 * WARPS + 32)
delta_recurrence_wide_kernel(const float* packed, float* state, long long slot_stride, float* o_out,
                             const int* cu_q_lens, const int* state_slots, int H, int D, int E) {
  extern __shared__ __align__(16) float dr_smem[];           // [DR_STAGES][DR_TOKENS][6 Dp]
  constexpr int Q = MAXR / 4;
  constexpr int Dp = LANES * MAXR;             // D and E, padded with zeros
  constexpr int COLS = 32 / LANES;             // a warp's columns side by side; CPT times as many in all
  constexpr int SV = 6 * Dp;                   // a token: w, b, u, k, r, v
  const int b = blockIdx.x, h = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_wait();                        // (launched in stream order; nothing is launched ahead of its end either)
  const int t0 = cu_q_lens[b], t1 = cu_q_lens[b + 1];
  if (t1 <= t0) return;
  const int groups = (t1 - t0 + DR_TOKENS - 1) / DR_TOKENS;
  if (Dp != D || Dp != E) {
    for (int i = threadIdx.x; i < DR_STAGES * DR_TOKENS * SV; i += blockDim.x) dr_smem[i] = 0.f;   // the padding stays 0
    __syncthreads();
  }
  if (warp == WARPS) {               // the copies
    const int PV = 5 * D + E;                  // a token's vectors of one head, as they are stored
    const bool wide = ((D | E) & 3) == 0;      // every vector starts on 16 bytes
    const long long token_step = (long long)H * PV;
    const float* base = packed + ((long long)t0 * H + h) * PV;
    auto fetch = [&](int g) {
      if (g < groups) {
        float* dst = dr_smem + (g % DR_STAGES) * DR_TOKENS * SV;
        const int n = min(DR_TOKENS, t1 - t0 - g * DR_TOKENS);
        const float* src = base + (long long)g * DR_TOKENS * token_step;
        for (int at = wide ? 4 * lane : lane; at < PV; at += wide ? 128 : 32) {
          const int vsel = at < 5 * D ? at / D : 5;
          float* to = dst + vsel * Dp + (at - vsel * D);
          const float* from = src + at;
          if (wide) {
            for (int i = 0; i < n; ++i, to += SV, from += token_step) __pipeline_memcpy_async(to, from, 16);
          } else {
            for (int i = 0; i < n; ++i, to += SV, from += token_step) __pipeline_memcpy_async(to, from, 4);
          }
        }
      }
      __pipeline_commit();                     // (an empty group past the end keeps the count)
    };
#pragma unroll
    for (int k = 0; k < DR_STAGES - 1; ++k) fetch(k);
    for (int g = 0; g < groups; ++g) {
      __pipeline_wait_prior(DR_STAGES - 2);    // group g has landed
      __syncthreads();                         // ... for everybody; everybody is done with group g - 1
      fetch(g + DR_STAGES - 1);                // into the stage of group g - 1
    }
    __pipeline_wait_prior(0);
    return;
  }
  const int s = lane % LANES;
  const int c = (blockIdx.z * WARPS + warp) * COLS * CPT + lane / LANES;       // this lane's columns: c, c + COLS, ...
  const long long slot = state_slots[b];
  const bool kept = slot != 0;       // slot 0 belongs to padding sequences: zero state, nothing stored
  float* S = state + slot * slot_stride + (long long)h * D * E;
  float st[CPT][MAXR];
#pragma unroll
  for (int j = 0; j < CPT; ++j)
#pragma unroll
    for (int ii = 0; ii < MAXR; ++ii) {
      const int i = (ii >> 2) * (4 * LANES) + s * 4 + (ii & 3);
      st[j][ii] = (kept && c + j * COLS < E && i < D) ? S[(long long)i * E + c + j * COLS] : 0.f;
    }
  // (volatile: the compiler would move the next token's loads behind the current one's work)
  auto load4 = [](unsigned at, float4& x) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(at));
  };
  const unsigned lane_at = (unsigned)__cvta_generic_to_shared(dr_smem) + s * 16;
  const unsigned v_at = (unsigned)__cvta_generic_to_shared(dr_smem) + (5 * Dp + c) * 4;
  auto read = [&](int at, DeltaToken<Q, CPT>& x) {
#pragma unroll
    for (int q = 0; q < Q; ++q) load4(lane_at + 4 * (at + q * 4 * LANES + 2 * Dp), x.u[q]);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      load4(lane_at + 4 * (at + q * 4 * LANES), x.w[q]);
      load4(lane_at + 4 * (at + q * 4 * LANES + 3 * Dp), x.k[q]);
    }
#pragma unroll
    for (int j = 0; j < CPT; ++j)
      asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x.v[j]) : "r"(v_at + 4 * (at + j * COLS)));
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      load4(lane_at + 4 * (at + q * 4 * LANES + Dp), x.b[q]);
      load4(lane_at + 4 * (at + q * 4 * LANES + 4 * Dp), x.r[q]);
    }
  };
  float* o_at = o_out + ((long long)(t0 - 1) * H + h) * E + c;    // where the token before the current one's output goes
  const long long o_step = (long long)H * E;
  float o_part[CPT] = {};                                    // this lane's part of it
  bool stores = false;                                       // there is a token before, and this lane stores its output
  auto store = [&](const float (&o)[CPT]) {
#pragma unroll
    for (int j = 0; j < CPT; ++j)
      if (stores && c + j * COLS < E) o_at[j * COLS] = o[j];
  };
  auto work = [&](const DeltaToken<Q, CPT>& x) {
    float dot[CPT], o[CPT];
#pragma unroll
    for (int j = 0; j < CPT; ++j) {
      float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        d0 = __fmaf_rn(x.u[q].x, st[j][q * 4 + 0], d0);
        d1 = __fmaf_rn(x.u[q].y, st[j][q * 4 + 1], d1);
        d2 = __fmaf_rn(x.u[q].z, st[j][q * 4 + 2], d2);
        d3 = __fmaf_rn(x.u[q].w, st[j][q * 4 + 3], d3);
      }
      dot[j] = __fadd_rn(__fadd_rn(d0, d1), __fadd_rn(d2, d3));
      o[j] = o_part[j];
    }
#pragma unroll
    for (int m = 1; m < LANES; m <<= 1) {
      float dx[CPT], ox[CPT];
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        dx[j] = __shfl_xor_sync(0xffffffffu, dot[j], m);
        ox[j] = __shfl_xor_sync(0xffffffffu, o[j], m);
      }
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        dot[j] = __fadd_rn(dot[j], dx[j]);
        o[j] = __fadd_rn(o[j], ox[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < CPT; ++j)
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        st[j][q * 4 + 0] = __fmaf_rn(x.k[q].x, x.v[j], __fmul_rn(x.w[q].x, st[j][q * 4 + 0]));
        st[j][q * 4 + 1] = __fmaf_rn(x.k[q].y, x.v[j], __fmul_rn(x.w[q].y, st[j][q * 4 + 1]));
        st[j][q * 4 + 2] = __fmaf_rn(x.k[q].z, x.v[j], __fmul_rn(x.w[q].z, st[j][q * 4 + 2]));
        st[j][q * 4 + 3] = __fmaf_rn(x.k[q].w, x.v[j], __fmul_rn(x.w[q].w, st[j][q * 4 + 3]));
      }
    store(o);
    o_at += o_step;
    stores = s == 0;
#pragma unroll
    for (int j = 0; j < CPT; ++j) {
      float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        st[j][q * 4 + 0] = __fmaf_rn(-x.b[q].x, dot[j], st[j][q * 4 + 0]);
        st[j][q * 4 + 1] = __fmaf_rn(-x.b[q].y, dot[j], st[j][q * 4 + 1]);
        st[j][q * 4 + 2] = __fmaf_rn(-x.b[q].z, dot[j], st[j][q * 4 + 2]);
        st[j][q * 4 + 3] = __fmaf_rn(-x.b[q].w, dot[j], st[j][q * 4 + 3]);
        o0 = __fmaf_rn(x.r[q].x, st[j][q * 4 + 0], o0);
        o1 = __fmaf_rn(x.r[q].y, st[j][q * 4 + 1], o1);
        o2 = __fmaf_rn(x.r[q].z, st[j][q * 4 + 2], o2);
        o3 = __fmaf_rn(x.r[q].w, st[j][q * 4 + 3], o3);
      }
      o_part[j] = __fadd_rn(__fadd_rn(o0, o1), __fadd_rn(o2, o3));
    }
  };

  for (int g = 0; g < groups; ++g) {
    __syncthreads();
    const int at = (g % DR_STAGES) * DR_TOKENS * SV;
    const int n = min(t1 - t0 - g * DR_TOKENS, DR_TOKENS);
    DeltaToken<Q, CPT> x, y;
    if (!NEXT || n < DR_TOKENS) {
#pragma unroll 1
      for (int i = 0; i < n; ++i) {
        read(at + i * SV, x);
        work(x);
      }
    } else {
      read(at, x);
#pragma unroll
      for (int i = 0; i < DR_TOKENS; i += 2) {
        read(at + (i + 1) * SV, y);
        work(x);
        if (i + 2 < DR_TOKENS) read(at + (i + 2) * SV, x);
        work(y);
      }
    }
  }
#pragma unroll
  for (int m = 1; m < LANES; m <<= 1)
#pragma unroll
    for (int j = 0; j < CPT; ++j) o_part[j] = __fadd_rn(o_part[j], __shfl_xor_sync(0xffffffffu, o_part[j], m));
  store(o_part);
#pragma unroll
  for (int j = 0; j < CPT; ++j)
#pragma unroll
    for (int ii = 0; ii < MAXR; ++ii) {
      const int i = (ii >> 2) * (4 * LANES) + s * 4 + (ii & 3);
      if (kept && c + j * COLS < E && i < D) S[(long long)i * E + c + j * COLS] = st[j][ii];
    }
}

// y[t, h, :] = o / sqrt(mean(o^2) + eps) * norm_w[h, :] * sigmoid(g[t, h, :])
// A warp per (token, head), 32 elements at a time: the sum of squares is the butterflies' over 32
// consecutive elements, added in index order.  CHUNKS: how many of them a row has at most (0: any
// number, read again behind the sum); the gate and the weight are asked for before the sum is made.
// SPLIT: the gate is split sums (decoded tokens), loaded four splits of all its elements at a time.
// (16 heads of 64, us: 2,048 tokens 8.5, blocks of D threads with a row each 34; 8 tokens of eight splits
// 2.2, an element's splits at a time 3.0, blocks of D threads 2.3.)
constexpr int OUT_WARPS = 8;
template <int CHUNKS, bool SPLIT>
__global__ void __launch_bounds__(OUT_WARPS * 32)
delta_output_kernel(const float* o, Source proj, const float* norm_w, void* out, int out_dtype, long long rows,
                    int H, int D, int R, float eps) {
  pdl_prologue();
  const long long row = (long long)blockIdx.x * OUT_WARPS + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const long long t = row / H;
  const int h = (int)(row - t * H), HD = H * D;
  const long long gate = t * (5 * HD + R) + 3 * HD + h * D;
  float ss = 0.f;
  if constexpr (CHUNKS > 0) {
    float x[CHUNKS], g[CHUNKS], w[CHUNKS];
#pragma unroll
    for (int j = 0; j < CHUNKS; ++j) {
      const int c = 32 * j + lane;
      x[j] = c < D ? o[row * D + c] : 0.f;
      w[j] = c < D ? norm_w[h * D + c] : 0.f;
    }
    if (SPLIT) {
      source_load_strided<CHUNKS, 4>(proj, gate, lane, 32, D, g);
    } else {
#pragma unroll
      for (int j = 0; j < CHUNKS; ++j) g[j] = 32 * j + lane < D ? source_load(proj, gate + 32 * j + lane) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < CHUNKS; ++j)
      if (32 * j < D) ss += warp_sum(x[j] * x[j]);
    const float rstd = 1.0f / sqrtf(ss / (float)D + eps);
#pragma unroll
    for (int j = 0; j < CHUNKS; ++j)
      if (32 * j + lane < D) store_as(out, out_dtype, row * D + 32 * j + lane, x[j] * rstd * w[j] * sigmoid_f32(g[j]));
  } else {
    for (int c0 = 0; c0 < D; c0 += 32) {
      const float x = c0 + lane < D ? o[row * D + c0 + lane] : 0.f;
      ss += warp_sum(x * x);
    }
    const float rstd = 1.0f / sqrtf(ss / (float)D + eps);
    for (int c = lane; c < D; c += 32)
      store_as(out, out_dtype, row * D + c,
               o[row * D + c] * rstd * norm_w[h * D + c] * sigmoid_f32(source_load(proj, gate + c)));
  }
}

// ---- gated delta rule: what goes in front of the recurrence and behind it ---------------------
// proj row (row_width elements): [q: G D | k: G D | v: H E | gate: H E | b: H | a: H | ...].  The
// convolutions' channels are the row's first CH = 2 G D + H E elements; cw [CH][taps] (the last
// tap is the current token's).  A sequence's inputs before the step's first token come from the
// tail of its state slot, [taps - 1][CH] floats at tail_at (oldest first); slot 0 has none (zeros).
__device__ __forceinline__ float conv_silu(const Source& proj, long long row_width, const float* cw,
                                           const float* tail, int CH, int taps, int t, int local, int ch) {
  float acc = 0.f;
  for (int j = 0; j < taps; ++j) {          // tap j reads the input taps - 1 - j tokens back
    const int back = taps - 1 - j;
    float x;
    if (back <= local) x = source_load(proj, (long long)(t - back) * row_width + ch);
    else x = tail != nullptr ? tail[(long long)(taps - 1 - (back - local)) * CH + ch] : 0.f;
    acc = __fmaf_rn(cw[(long long)ch * taps + j], x, acc);
  }
  return acc * sigmoid_f32(acc);
}

// One block per (token, value head): packed [T][H][5 D + E] = w (the decay in every row), g beta u,
// u, beta u, q (unit, times D^-1/2), v; u the unit key.
__global__ void gated_delta_prepare_kernel(Source proj, long long row_width, const float* cw, const float* a_log,
                                           const float* dt_bias, const float* state, long long slot_stride,
                                           long long tail_at, const int* token_seq, const int* cu_q_lens,
                                           const int* state_slots, float* packed, int H, int G, int D, int E,
                                           int taps, float key_eps) {
  __shared__ float scratch[32];
  pdl_prologue(proj.p);
  const int t = blockIdx.x, h = blockIdx.y, c = threadIdx.x;
  const int g = h / (H / G);
  const int CH = 2 * G * D + H * E;
  const int b = token_seq[t];
  const int local = t - cu_q_lens[b];
  const long long slot = state_slots[b];
  const float* tail = slot != 0 ? state + slot * slot_stride + tail_at : nullptr;
  float q = 0.f, k = 0.f, v = 0.f;
  if (c < D) {
    q = conv_silu(proj, row_width, cw, tail, CH, taps, t, local, g * D + c);
    k = conv_silu(proj, row_width, cw, tail, CH, taps, t, local, G * D + g * D + c);
  }
  if (c < E) v = conv_silu(proj, row_width, cw, tail, CH, taps, t, local, 2 * G * D + h * E + c);
  const float qq = block_sum(q * q, scratch);
  const float kk = block_sum(k * k, scratch);
  const long long row = (long long)t * row_width;
  const float beta = sigmoid_f32(source_load(proj, row + CH + (long long)H * E + h));
  const float z = __fadd_rn(source_load(proj, row + CH + (long long)H * E + H + h), dt_bias[h]);
  const float softplus = z > 20.f ? z : log1pf(expf(z));
  const float decay = expf(-expf(a_log[h]) * softplus);
  float* out = packed + ((long long)t * H + h) * (5 * D + E);
  if (c < D) {
    const float u = k / sqrtf(kk + key_eps);
    out[c] = decay;
    out[D + c] = decay * beta * u;
    out[2 * D + c] = u;
    out[3 * D + c] = beta * u;
    out[4 * D + c] = q / sqrtf(qq + key_eps) * rsqrtf((float)D);
  }
  if (c < E) out[5 * D + c] = v;
}

// y[t, h, :] = o / sqrt(mean(o^2) + eps) * norm_w[:] * silu(gate[t, h, :]); the weight is shared by the heads
__global__ void gated_delta_output_kernel(const float* o, Source proj, long long row_width, long long gate_col,
                                          const float* norm_w, void* out, int out_dtype, int H, int E, float eps) {
  __shared__ float scratch[32];
  pdl_prologue(o, proj.p);
  const int t = blockIdx.x, h = blockIdx.y, c = threadIdx.x;
  const long long at = ((long long)t * H + h) * E + c;
  const float x = c < E ? o[at] : 0.f;
  const float ss = block_sum(x * x, scratch);
  if (c < E) {
    const float rstd = 1.0f / sqrtf(ss / (float)E + eps);
    const float g = source_load(proj, (long long)t * row_width + gate_col + (long long)h * E + c);
    store_as(out, out_dtype, at, x * rstd * norm_w[c] * (g * sigmoid_f32(g)));
  }
}

template <int MAXR, int DR_STAGES>
static int launch_recurrence(const float* packed, float* state, long long slot_stride, float* o_out,
                             const int* cu_q_lens, const int* state_slots, int B, int H, int D, int E, cudaStream_t st) {
  const int Dp = (D + 15) / 16 * 16, Ep = (E + 15) / 16 * 16;
  const size_t smem = sizeof(float) * 4 * DR_STAGES * (5 * Dp + Ep);   // 48 KB at D = E = 64, 72 at 128, 96 at 256
  static DeviceOnce once;
  if (smem > 48 * 1024 && !once.done()) {
    if (cudaFuncSetAttribute(delta_recurrence_kernel<MAXR, DR_STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             100 * 1024) != cudaSuccess)
      return DIB_LAUNCH_FAILED;
    once.mark();
  }
  dib_launch(delta_recurrence_kernel<MAXR, DR_STAGES>, dim3(B, H, (E + 31) / 32), dim3(128), smem, st, packed, state,
             slot_stride, o_out, cu_q_lens, state_slots, H, D, E);
  DIB_CHECK_LAUNCH();
  return DIB_OK;
}

template <int MAXR, int LANES, int CPT, int WARPS, int DR_TOKENS, int DR_STAGES, bool NEXT>
static int launch_recurrence_wide(const float* packed, float* state, long long slot_stride, float* o_out,
                                  const int* cu_q_lens, const int* state_slots, int B, int H, int D, int E,
                                  cudaStream_t st) {
  constexpr int COLUMNS = 32 / LANES * CPT * WARPS;        // a block's
  constexpr size_t smem = sizeof(float) * DR_STAGES * DR_TOKENS * 6 * LANES * MAXR;    // 48 KB for 64, 96 for 128 and 256
  auto* kernel = &delta_recurrence_wide_kernel<MAXR, LANES, CPT, WARPS, DR_TOKENS, DR_STAGES, NEXT>;
  static DeviceOnce once;
  if (!once.done()) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return DIB_LAUNCH_FAILED;
    once.mark();
  }
  // Launched in plain stream order, not ahead of its predecessor's end: blocks that are placed
  // while the kernel before still fills the GPU land several to an SM on the SMs that happen to
  // be free, and a long chain of dependent instructions then shares its scheduler for the whole
  // kernel.
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(B, H, (E + COLUMNS - 1) / COLUMNS);
  cfg.blockDim = dim3(32 * WARPS + 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchKernelEx(&cfg, kernel, packed, state, slot_stride, o_out, cu_q_lens, state_slots, H, D, E);
  DIB_CHECK_LAUNCH();
  return DIB_OK;
}

extern "C" {

int dib_delta_prepare(const void* proj, int kind, int splits, long long stride, const void* w2t, int w_dtype,
                      const float* w0, const float* a_bias, float* packed, int T_, int H, int D, int R,
                      float decay_scale, float key_eps, cudaStream_t st) {
  if (T_ == 0) return DIB_OK;
  if (H < 1 || H > 65535 || D < 1 || D > 1024 || R < 0 || R > 8192) return DIB_BAD_SIZE;
  if (w_dtype != 0 && w_dtype != 1) return DIB_BAD_DTYPE;
  const Source src = make_source(proj, kind, splits, stride);
  auto go = [&](auto tokens, auto* kernel) {
    constexpr int N = decltype(tokens)::value;
    dib_launch(kernel, dim3(ceil_div_host(T_, N), H), dim3((D + 31) / 32 * 32), 0, st, src, w2t, w0, a_bias, packed, T_,
               H, D, R, decay_scale, key_eps);
  };
  auto stored = [&](auto tokens) {
    constexpr int N = decltype(tokens)::value;
    go(tokens, kind == 1 ? (w_dtype == 1 ? &delta_prepare_kernel<N, 1, 1> : &delta_prepare_kernel<N, 1, 0>)
                         : (w_dtype == 1 ? &delta_prepare_kernel<N, 0, 1> : &delta_prepare_kernel<N, 0, 0>));
  };
  const std::integral_constant<int, 1> one;
  if (kind != 1 && splits > 1) go(one, w_dtype == 1 ? &delta_prepare_kernel<1, 2, 1> : &delta_prepare_kernel<1, 2, 0>);
  // (heads of more than 256: a block's registers do not reach for the values of several tokens)
  else if (D > 256) stored(one);
  else if (T_ < PREP_FOUR_FROM) stored(std::integral_constant<int, 2>{});
  else stored(std::integral_constant<int, 4>{});
  DIB_CHECK_LAUNCH();
  return DIB_OK;
}

// state: float32 rows of slot_stride elements, a slot's first H * D * E the heads' states [H, D, E];
// sequence b of the step owns tokens cu_q_lens[b] .. cu_q_lens[b+1]-1 and the state slot
// state_slots[b].  Slot 0 is no request's: a sequence on it starts from a zero state and leaves none.
// packed [T][H][5 D + E].
// form 1: a column's rows over 16 lanes (for steps of few sequences with many tokens), 0: over 4.
int dib_delta_recurrence(const float* packed, float* state, long long slot_stride, float* o_out,
                         const int* cu_q_lens, const int* state_slots, int B, int H, int D, int E, int form,
                         cudaStream_t st) {
  if (B == 0) return DIB_OK;
  if (H < 1 || H > 65535 || D < 1 || D > 256 || E < 1 || E > 256) return DIB_BAD_SIZE;
  const int big = D > E ? D : E;       // (the staging's pieces are counted for the larger of the two)
#define DIB_DR(F, ...) return F<__VA_ARGS__>(packed, state, slot_stride, o_out, cu_q_lens, state_slots, B, H, D, E, st)
  if (form == 1) {
    if (big <= 64) DIB_DR(launch_recurrence_wide, 4, 16, 1, 4, 16, 2, true);
    if (big <= 128) DIB_DR(launch_recurrence_wide, 8, 16, 2, 4, 16, 2, true);
    DIB_DR(launch_recurrence_wide, 16, 16, 2, 4, 8, 2, false);
  }
  if (big <= 64) DIB_DR(launch_recurrence, 16, 8);
  if (big <= 128) DIB_DR(launch_recurrence, 32, 6);
  DIB_DR(launch_recurrence, 64, 4);
#undef DIB_DR
}

int dib_delta_output(const float* o, const void* proj, int kind, int splits, long long stride,
                     const float* norm_w, void* out, int out_dtype, int T_, int H, int D, int R, float eps,
                     cudaStream_t st) {
  if (T_ == 0) return DIB_OK;
  if (H < 1 || H > 65535 || D < 1 || D > 1024) return DIB_BAD_SIZE;
  if (out_dtype != 0 && out_dtype != 1) return DIB_BAD_DTYPE;
  const long long rows = (long long)T_ * H;
  auto* kernel = kind != 1 && splits > 1
                     ? (D <= 64 ? &delta_output_kernel<2, true> : D <= 128 ? &delta_output_kernel<4, true> : &delta_output_kernel<0, true>)
                     : (D <= 64 ? &delta_output_kernel<2, false> : D <= 128 ? &delta_output_kernel<4, false> : &delta_output_kernel<0, false>);
  dib_launch(kernel, dim3(ceil_div_host(rows, OUT_WARPS)), dim3(OUT_WARPS * 32), 0, st, o,
             make_source(proj, kind, splits, stride), norm_w, out, out_dtype, rows, H, D, R, eps);
  DIB_CHECK_LAUNCH();
  return DIB_OK;
}

int dib_gated_delta_prepare(const void* proj, int kind, int splits, long long stride, long long row_width,
                            const float* cw, const float* a_log, const float* dt_bias, const float* state,
                            long long slot_stride, long long tail_at, const int* token_seq, const int* cu_q_lens,
                            const int* state_slots, float* packed, int T_, int H, int G, int D, int E, int taps,
                            float key_eps, cudaStream_t st) {
  if (T_ == 0) return DIB_OK;
  if (H < 1 || H > 65535 || G < 1 || H % G || D < 1 || D > 1024 || E < 1 || E > 1024 || taps < 1 || taps > 64)
    return DIB_BAD_SIZE;
  const int width = D > E ? D : E;
  dib_launch(gated_delta_prepare_kernel, dim3(T_, H), dim3((width + 31) / 32 * 32), 0, st,
             make_source(proj, kind, splits, stride), row_width, cw, a_log, dt_bias, state, slot_stride, tail_at,
             token_seq, cu_q_lens, state_slots, packed, H, G, D, E, taps, key_eps);
  DIB_CHECK_LAUNCH();
  return DIB_OK;
}

// The output rows, and then (B sequences) the convolutions' tails moved on by the step's tokens.
int dib_gated_delta_output(const float* o, const void* proj, int kind, int splits, long long stride,
                           long long row_width, const float* norm_w, void* out, int out_dtype, float* state,
                           long long slot_stride, long long tail_at, const int* cu_q_lens, const int* state_slots,
                           int T_, int B, int H, int G, int D, int E, int taps, float eps, cudaStream_t st) {
  if (T_ == 0) return DIB_OK;
  if (H < 1 || H > 65535 || G < 1 || E < 1 || E > 1024 || taps < 1) return DIB_BAD_SIZE;
  if (out_dtype != 0 && out_dtype != 1) return DIB_BAD_DTYPE;
  const Source src = make_source(proj, kind, splits, stride);
  const int CH = 2 * G * D + H * E;
  dib_launch(gated_delta_output_kernel, dim3(T_, H), dim3((E + 31) / 32 * 32), 0, st, o, src, row_width,
             (long long)CH, norm_w, out, out_dtype, H, E, eps);
  DIB_CHECK_LAUNCH();
  if (taps > 1 && B > 0) {
    dib_launch(conv_tail_update_kernel, dim3(B), dim3(256), 0, st, src, row_width, 0ll, (const float*)nullptr, state,
               slot_stride, tail_at, cu_q_lens, state_slots, CH, taps);
    DIB_CHECK_LAUNCH();
  }
  return DIB_OK;
}

}  // extern "C"

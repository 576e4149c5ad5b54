// Sampling kernels over float32 logits [R, V]: argmax (lowest index wins ties)
// and temperature sampling by position-seeded Gumbel-max.
//
// Gumbel-max: p = softmax(logits / temperature); token = argmax over kept ids of
// log(p + 1e-10) + g(seed, pos, id), with g = -log(-log(u + 1e-10) + 1e-10) and u
// the low 24 bits of a 64-bit wrap-around hash of (seed, pos, id) divided by
// 2^24.  The noise is a pure function of (seed, position of the generated token,
// vocabulary id), so a draw does not depend on the batch.  Rows with
// temperature <= 0 take the argmax.  `keep` (optional, uint8 [R, V]) masks ids
// dropped by top-k / top-p.
#include "common.cuh"

namespace {

struct Best {
  float v;
  int i;
};

__device__ __forceinline__ Best better(Best a, Best b) {
  // larger value wins; equal values: lower index wins
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}

__device__ __forceinline__ Best block_best(Best b, Best* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Best other;
    other.v = __shfl_xor_sync(0xffffffffu, b.v, o);
    other.i = __shfl_xor_sync(0xffffffffu, b.i, o);
    b = better(b, other);
  }
  __syncthreads();
  if (lane == 0) scratch[warp] = b;
  __syncthreads();
  Best r = scratch[0];
  for (int w = 1; w < nwarps; ++w) r = better(r, scratch[w]);
  return r;
}

__device__ __forceinline__ float block_max(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float r = scratch[0];
  for (int w = 1; w < nwarps; ++w) r = fmaxf(r, scratch[w]);
  return r;
}

constexpr int INT_MAX_ = 0x7fffffff;

__global__ void argmax_kernel(const float* __restrict__ logits, int* __restrict__ out, int V) {
  pdl_prologue(logits);
  __shared__ Best scratch[32];
  const float* row = logits + (size_t)blockIdx.x * V;
  Best b{-INFINITY, INT_MAX_};
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    Best c{row[i], i};
    b = better(b, c);
  }
  b = block_best(b, scratch);
  if (threadIdx.x == 0) out[blockIdx.x] = b.i == INT_MAX_ ? 0 : b.i;
}

// Two-stage argmax for wide rows: a row is cut into chunks of ARGMAX_CHUNK ids,
// one block per (row, chunk) writes its best (value, index); a second kernel picks
// the best chunk.  Ties go to the lowest index in both stages.
constexpr int ARGMAX_CHUNK = 4096;

__global__ void argmax_partial_kernel(const float* __restrict__ logits, float* __restrict__ pv,
                                      int* __restrict__ pi, int V, int chunks) {
  pdl_prologue(logits);
  __shared__ Best scratch[32];
  const int r = blockIdx.y, c = blockIdx.x;
  const float* row = logits + (size_t)r * V;
  const int lo = c * ARGMAX_CHUNK, hi = min(V, lo + ARGMAX_CHUNK);
  Best b{-INFINITY, INT_MAX_};
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) b = better(b, Best{row[i], i});
  b = block_best(b, scratch);
  if (threadIdx.x == 0) {
    pv[(size_t)r * chunks + c] = b.v;
    pi[(size_t)r * chunks + c] = b.i;
  }
}

__global__ void argmax_final_kernel(const float* __restrict__ pv, const int* __restrict__ pi,
                                    int* __restrict__ out, int chunks) {
  pdl_prologue(pv, pi);
  __shared__ Best scratch[32];
  const int r = blockIdx.x;
  Best b{-INFINITY, INT_MAX_};
  for (int c = threadIdx.x; c < chunks; c += blockDim.x)
    b = better(b, Best{pv[(size_t)r * chunks + c], pi[(size_t)r * chunks + c]});
  b = block_best(b, scratch);
  if (threadIdx.x == 0) out[r] = b.i == INT_MAX_ ? 0 : b.i;
}

__device__ __forceinline__ float seeded_gumbel(long long seed, long long pos, int col) {
  const unsigned long long step =
      ((unsigned long long)seed * 19349663ull) ^ ((unsigned long long)pos * 73856093ull);
  const unsigned long long hashed =
      (step * 8589934591ull) ^ ((unsigned long long)col * 479001599ull);
  const float u = (float)(unsigned)(hashed & 0xffffffull) / 16777216.0f;
  return -logf(-logf(u + 1e-10f) + 1e-10f);
}

__global__ void gumbel_sample_kernel(const float* __restrict__ logits,
                                     const float* __restrict__ temperatures,
                                     const long long* __restrict__ seeds,
                                     const long long* __restrict__ sample_pos,
                                     const unsigned char* __restrict__ keep,
                                     int* __restrict__ out, int V) {
  pdl_prologue(logits, temperatures, seeds, sample_pos, keep);
  __shared__ Best bscratch[32];
  __shared__ float fscratch[32];
  const int r = blockIdx.x;
  const float* row = logits + (size_t)r * V;
  const float temp = temperatures[r];
  if (temp <= 0.f) {
    Best b{-INFINITY, INT_MAX_};
    for (int i = threadIdx.x; i < V; i += blockDim.x) b = better(b, Best{row[i], i});
    b = block_best(b, bscratch);
    if (threadIdx.x == 0) out[r] = b.i == INT_MAX_ ? 0 : b.i;
    return;
  }
  float mx = -INFINITY;
  for (int i = threadIdx.x; i < V; i += blockDim.x) mx = fmaxf(mx, row[i] / temp);
  mx = block_max(mx, fscratch);
  float sum = 0.f;
  for (int i = threadIdx.x; i < V; i += blockDim.x) sum += expf(row[i] / temp - mx);
  sum = block_sum(sum, fscratch);
  const long long seed = seeds[r], pos = sample_pos[r];
  const unsigned char* krow = keep ? keep + (size_t)r * V : nullptr;
  Best b{-INFINITY, INT_MAX_};
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    if (krow && !krow[i]) continue;
    const float p = expf(row[i] / temp - mx) / sum;
    const float score = logf(p + 1e-10f) + seeded_gumbel(seed, pos, i);
    b = better(b, Best{score, i});
  }
  b = block_best(b, bscratch);
  if (threadIdx.x == 0) out[r] = b.i == INT_MAX_ ? 0 : b.i;
}
// Wide rows in chunks of ARGMAX_CHUNK ids, one block per (row, chunk), three kernels:
// the chunk's maximum of logits / temperature and its sum of exponentials against that
// maximum; then, with the row's maximum and sum put together from the chunks' in chunk
// order (a row's normaliser never depends on the batch), the chunk's best score; then
// the best chunk (argmax_final_kernel).
//
// The chunk lies in registers, 16 ids a thread, loaded before anything else is waited for.
// These kernels are bound by instructions, not by the logits (39 MB for 64 rows of 151,936
// stay in L2): a probability costs two divisions and an exponential, a score three more
// logarithms.  So each of them first looks at a cheap value with a margin (log2 of the
// probability by one FMA, an upper bound of the score by one logarithm more) and forms the
// exact one, always by the same expressions, only where that can matter.
constexpr int SAMPLE_THREADS = 256;
constexpr int PER_THREAD = ARGMAX_CHUNK / SAMPLE_THREADS;

__device__ __forceinline__ void load_chunk(const float* __restrict__ row, int lo, int hi, float (&x)[PER_THREAD]) {
#pragma unroll
  for (int j = 0; j < PER_THREAD; ++j) {
    const int i = lo + threadIdx.x + j * SAMPLE_THREADS;
    x[j] = i < hi ? row[i] : -INFINITY;
  }
}

// top-k / top-p without a sort.  In the order of a descending sort a token stays when
// its rank is below k and the probability mass before it is at most top_p (rank 0 always
// stays).  Rank and mass before are both non-increasing in the token's probability, so
// the kept set is {p >= t} for one threshold t: found by a radix descent over the 31
// bits of the probability (it has no sign), 10, 11 and 10 bits a pass, with a histogram of
// counts and of masses per pass.  Masses are added as 40-bit fixed point, so that the order
// of the additions (atomics) cannot change a bit.  Tokens that tie with the threshold all
// stay (a sort would keep some of them).  The first two passes have a block per chunk of a
// row; the block that is last to add its histogram to the row's works out the row's bits and
// leaves them for the next pass.  The first forms every probability; the second only those
// whose log2 may lie in the first's bin, and lists the bin's probabilities; the third is a
// block a row over that list.  A flat row has more tokens in one bin than the list holds:
// THIRD_BLOCKS blocks go over the row again then and add to a histogram as the others do (8 such
// rows of 151,936: the whole draw 91 us; by one block a row 398 us).
// (Four passes of 8 bits that formed every probability again, added up a warp's equal bins
// by matching lanes and chained the chunks' normalisers in every thread: 69 us each, and
// the pick 68 us; with 64 rows of 151,936, 38 of them filtered, the whole draw 318 us.  Three
// passes over the chunks, each of whose blocks works out the pass before: 122 us; so
// 104 us.)
constexpr float MASS_ONE = 1099511627776.0f;     // 2^40
constexpr int FILTER_BINS0 = 1024, FILTER_BINS1 = 2048, FILTER_BINS2 = 1024;      // of the passes
constexpr int FILTER_SHIFT0 = 21, FILTER_SHIFT1 = 10;
constexpr int FILTER_BINS = FILTER_BINS0 + FILTER_BINS1;       // a row's in global memory
static_assert(FILTER_BINS2 <= FILTER_BINS0, "the third pass may use the first one's histogram");
constexpr int FILTER_LIST = 16384;                             // probabilities a row's list holds
constexpr int FILTER_ROWS = 512;                               // filtered rows at a time: 52 MB of scratch
constexpr int THIRD_BLOCKS = 8;                                // blocks a row of the third pass

struct FilterState {
  unsigned long long cnt_above, mass_above;   // tokens (and their mass) above the chosen bins
  unsigned prefix;                            // the threshold's bits found so far
  unsigned pad;
};
// a row's counters: blocks that have added to the first, the second and the third histogram, listed probabilities
enum { MARK_FIRST = 0, MARK_SECOND = 1, MARK_LISTED = 2, MARK_THIRD = 3, ROW_MARKS = 4 };

__global__ void __launch_bounds__(SAMPLE_THREADS)
gumbel_stats_kernel(const float* __restrict__ logits, const float* __restrict__ temperatures,
                    float* __restrict__ cmax, float* __restrict__ csum, unsigned* __restrict__ hist_cnt,
                    unsigned long long* __restrict__ hist_mass, unsigned* __restrict__ marks, int V, int chunks) {
  pdl_prologue(logits, temperatures);
  __shared__ float fscratch[32];
  const int r = blockIdx.y, c = blockIdx.x;
  // the row's top-k / top-p histograms start from zero: the blocks of the row share the zeroing
  if (hist_cnt != nullptr) {
    for (int e = c * SAMPLE_THREADS + threadIdx.x; e < FILTER_BINS; e += chunks * SAMPLE_THREADS) {
      hist_cnt[(size_t)r * FILTER_BINS + e] = 0u;
      hist_mass[(size_t)r * FILTER_BINS + e] = 0ull;
    }
    if (c == 0 && threadIdx.x < ROW_MARKS) marks[(size_t)r * ROW_MARKS + threadIdx.x] = 0u;
  }
  const float temp = temperatures[r];
  if (temp <= 0.f) return;     // a greedy row needs no normaliser
  const int lo = c * ARGMAX_CHUNK, hi = min(V, lo + ARGMAX_CHUNK);
  float x[PER_THREAD];
  load_chunk(logits + (size_t)r * V, lo, hi, x);
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < PER_THREAD; ++j) mx = fmaxf(mx, x[j]);
  // (rounding keeps order: the largest quotient is the quotient of the largest)
  mx = block_max(mx, fscratch) / temp;
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < PER_THREAD; ++j)
    if (lo + (int)threadIdx.x + j * SAMPLE_THREADS < hi) sum += expf(x[j] / temp - mx);
  sum = block_sum(sum, fscratch);
  if (mx == -INFINITY) sum = 0.f;      // (a chunk of ids that are all out adds nothing to its row)
  if (threadIdx.x == 0) {
    cmax[(size_t)r * chunks + c] = mx;
    csum[(size_t)r * chunks + c] = sum;
  }
}

// The row's maximum and sum of exponentials from its chunks', in chunk order: every
// kernel that needs a probability forms it from these two, with the same expression, so
// all of them see the same bits.  The exponentials are taken by the threads side by side.
struct NormaliserScratch {
  float f[32], e[SAMPLE_THREADS], s[SAMPLE_THREADS];
};
__device__ __forceinline__ void row_normaliser(const float* __restrict__ cmax, const float* __restrict__ csum, int r,
                                               int chunks, NormaliserScratch& sc, float& mx, float& sum) {
  const float* cm = cmax + (size_t)r * chunks;
  const float* cs = csum + (size_t)r * chunks;
  mx = -INFINITY;
  for (int k = threadIdx.x; k < chunks; k += SAMPLE_THREADS) mx = fmaxf(mx, cm[k]);
  mx = block_max(mx, sc.f);
  sum = 0.f;
  for (int base = 0; base < chunks; base += SAMPLE_THREADS) {
    __syncthreads();
    if (base + (int)threadIdx.x < chunks) {
      sc.e[threadIdx.x] = expf(cm[base + threadIdx.x] - mx);
      sc.s[threadIdx.x] = cs[base + threadIdx.x];
    }
    __syncthreads();
    const int n = min(SAMPLE_THREADS, chunks - base);
#pragma unroll 8
    for (int k = 0; k < n; ++k) sum = __fmaf_rn(sc.s[k], sc.e[k], sum);
  }
}
__device__ __forceinline__ float row_probability(float logit, float temp, float mx, float sum) {
  return expf(logit / temp - mx) / sum;
}

// log2 of a probability up to `margin`, by one FMA; not usable (`ok` false) at temperatures
// and maxima whose products leave the range of float32.
struct Estimate {
  float a, c, margin;
  bool ok;
  __device__ __forceinline__ Estimate(float temp, float mx, float sum) {
    a = 1.4426950408889634f / temp;
    c = fmaf(mx, 1.4426950408889634f, log2f(sum));
    ok = fabsf(a) < 1e30f && fabsf(c) < 1e30f;
    // roundings of the quotient, of a and of the FMA: a few 2^-24 of |c| + 150, wherever the
    // probability is not zero
    margin = 1e-3f + 1e-6f * fabsf(c);
  }
  __device__ __forceinline__ float log2p(float logit) const { return fmaf(logit, a, -c); }
};
// bounds of log2p for probabilities whose bits lie in [first, last]; denormal ones have no
// relative accuracy and get no tight bound
__device__ __forceinline__ float lower_bound(unsigned first, const Estimate& e) {
  return first < 0x01000000u ? -INFINITY : log2f(__uint_as_float(first)) - e.margin;
}
__device__ __forceinline__ float upper_bound(unsigned last, const Estimate& e) {
  return last < 0x01000000u ? -100.f : log2f(__uint_as_float(last)) + e.margin;
}

// The whole block: the state after pass `pass`, from the state before it and its histogram.
struct DescendScratch {
  unsigned long long m[8];
  unsigned c[8];
  int chosen[8];
  FilterState st;
};
// (SHARED: the histograms lie in shared memory)
template <int BINS, bool SHARED = false>
__device__ __forceinline__ FilterState filter_descend(const unsigned* hist_cnt, const unsigned long long* hist_mass,
                                                      FilterState st, int shift, unsigned long long k,
                                                      unsigned long long P, DescendScratch& sc) {
  constexpr int B = BINS / SAMPLE_THREADS;       // a thread's bins
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned c[B], csum = 0u;
  unsigned long long m[B], msum = 0ull;
#pragma unroll
  for (int j = 0; j < B; ++j) {
    c[j] = SHARED ? hist_cnt[threadIdx.x * B + j] : __ldcg(hist_cnt + threadIdx.x * B + j);
    m[j] = SHARED ? hist_mass[threadIdx.x * B + j] : __ldcg(hist_mass + threadIdx.x * B + j);
    csum += c[j];
    msum += m[j];
  }
  // counts and masses of the bins of higher threads (an exclusive suffix sum)
  unsigned c_run = csum;
  unsigned long long m_run = msum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned c_up = __shfl_down_sync(0xffffffffu, c_run, o);
    const unsigned long long m_up = __shfl_down_sync(0xffffffffu, m_run, o);
    if (lane + o < 32) {
      c_run += c_up;
      m_run += m_up;
    }
  }
  __syncthreads();
  if (lane == 0) {
    sc.c[warp] = c_run;
    sc.m[warp] = m_run;
  }
  __syncthreads();
  unsigned long long ca = st.cnt_above + c_run - csum, ma = st.mass_above + m_run - msum;
  for (int w = warp + 1; w < SAMPLE_THREADS / 32; ++w) {
    ca += sc.c[w];
    ma += sc.m[w];
  }
  // this thread's bins from the highest down: the lowest non-empty bin that is entered
  // while fewer than k tokens, weighing at most P, lie above it
  int best = BINS;
  unsigned long long best_ca = 0ull, best_ma = 0ull;
#pragma unroll
  for (int j = B - 1; j >= 0; --j) {
    if (c[j] != 0u && ca < k && ma <= P) {
      best = threadIdx.x * B + j;
      best_ca = ca;
      best_ma = ma;
    }
    ca += c[j];
    ma += m[j];
  }
  const int wbest = __reduce_min_sync(0xffffffffu, best);
  if (lane == 0) sc.chosen[warp] = wbest;
  __syncthreads();
  int chosen = sc.chosen[0];
#pragma unroll
  for (int w = 1; w < SAMPLE_THREADS / 32; ++w) chosen = min(chosen, sc.chosen[w]);
  // (an empty histogram, chosen == BINS, cannot happen for a row that is filtered: bin 0 then)
  if (best == chosen && best < BINS) sc.st = FilterState{best_ca, best_ma, st.prefix | ((unsigned)best << shift), 0u};
  if (chosen == BINS && threadIdx.x == 0) sc.st = FilterState{0ull, 0ull, st.prefix, 0u};
  __syncthreads();
  return sc.st;
}
// Has every block of the row added to its histogram (this one just has)?  The same answer in all threads.
__device__ __forceinline__ bool last_of_row(unsigned* mark, int chunks, bool* flag) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) *flag = atomicAdd(mark, 1u) == (unsigned)chunks - 1u;
  __syncthreads();
  if (*flag) __threadfence();
  return *flag;
}
// One token's probability into histograms of `bins` counts and masses in halves of 20 bits, whose sums over a
// chunk fit 32 bits; every lane of the warp calls.  32 tokens of one bin (a flat row, a tail that underflows) are
// one addition.
__device__ __forceinline__ void count_token(float p, unsigned bin, bool in, unsigned* cnt, unsigned* low, unsigned* high) {
  const unsigned long long m = (unsigned long long)(p * MASS_ONE);
  const unsigned first = __shfl_sync(0xffffffffu, bin, 0);
  if (__all_sync(0xffffffffu, in && bin == first)) {
    const unsigned l = __reduce_add_sync(0xffffffffu, (unsigned)(m & 0xfffffull));
    const unsigned h = __reduce_add_sync(0xffffffffu, (unsigned)(m >> 20));
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&cnt[bin], 32u);
      atomicAdd(&low[bin], l);
      atomicAdd(&high[bin], h);
    }
  } else if (in) {
    atomicAdd(&cnt[bin], 1u);
    atomicAdd(&low[bin], (unsigned)(m & 0xfffffull));
    atomicAdd(&high[bin], (unsigned)(m >> 20));
  }
}
template <int BINS>
__device__ __forceinline__ void add_histogram(const unsigned* cnt, const unsigned* low, const unsigned* high,
                                              unsigned* __restrict__ hist_cnt,
                                              unsigned long long* __restrict__ hist_mass) {
  for (int b = threadIdx.x; b < BINS; b += SAMPLE_THREADS)
    if (cnt[b] != 0u) {
      atomicAdd(&hist_cnt[b], cnt[b]);
      atomicAdd(&hist_mass[b], ((unsigned long long)high[b] << 20) + low[b]);
    }
}
// what a row asks for: fewer than k tokens above a kept one, weighing at most P
struct FilterLimits {
  unsigned long long k, P;
  __device__ __forceinline__ FilterLimits(long long top_k, float top_p, int V)
      : k(top_k > 0 ? (unsigned long long)top_k : (unsigned long long)V + 1),
        P(top_p >= 1.0f ? ~0ull : (unsigned long long)(top_p * MASS_ONE)) {}
};

__device__ __forceinline__ bool row_is_filtered(float temp, long long top_k, float top_p) {
  return temp > 0.f && (top_k > 0 || top_p < 1.0f);
}

// states: [2][R], what the first and the second pass find
__global__ void __launch_bounds__(SAMPLE_THREADS)
filter_first_kernel(const float* __restrict__ logits, const float* __restrict__ temperatures,
                    const long long* __restrict__ top_ks, const float* __restrict__ top_ps,
                    const float* __restrict__ cmax, const float* __restrict__ csum, unsigned* hist_cnt,
                    unsigned long long* hist_mass, FilterState* __restrict__ states, float2* __restrict__ norms,
                    unsigned* marks, int V, int chunks) {
  pdl_prologue(logits, temperatures, top_ks, top_ps, cmax, csum);
  __shared__ unsigned s_cnt[FILTER_BINS0], s_low[FILTER_BINS0], s_high[FILTER_BINS0];
  __shared__ NormaliserScratch nsc;
  __shared__ DescendScratch dsc;
  __shared__ bool s_last;
  const int r = blockIdx.y, c = blockIdx.x;
  const float temp = temperatures[r];
  const long long top_k = top_ks[r];
  const float top_p = top_ps[r];
  float mx, sum;
  if (!row_is_filtered(temp, top_k, top_p)) {
    if (c == 0 && temp > 0.f) {                    // (the pick reads every row's normaliser)
      row_normaliser(cmax, csum, r, chunks, nsc, mx, sum);
      if (threadIdx.x == 0) norms[r] = make_float2(mx, sum);
    }
    return;
  }
  const int lo = c * ARGMAX_CHUNK, hi = min(V, lo + ARGMAX_CHUNK);
  float x[PER_THREAD];
  load_chunk(logits + (size_t)r * V, lo, hi, x);
  for (int b = threadIdx.x; b < FILTER_BINS0; b += SAMPLE_THREADS) s_cnt[b] = s_low[b] = s_high[b] = 0u;
  row_normaliser(cmax, csum, r, chunks, nsc, mx, sum);
  if (c == 0 && threadIdx.x == 0) norms[r] = make_float2(mx, sum);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < PER_THREAD; ++j) {
    const float p = row_probability(x[j], temp, mx, sum);
    count_token(p, (__float_as_uint(p) >> FILTER_SHIFT0) & (FILTER_BINS0 - 1),
                lo + (int)threadIdx.x + j * SAMPLE_THREADS < hi, s_cnt, s_low, s_high);
  }
  __syncthreads();
  hist_cnt += (size_t)r * FILTER_BINS;
  hist_mass += (size_t)r * FILTER_BINS;
  add_histogram<FILTER_BINS0>(s_cnt, s_low, s_high, hist_cnt, hist_mass);
  if (last_of_row(&marks[(size_t)r * ROW_MARKS + MARK_FIRST], chunks, &s_last)) {
    const FilterLimits lim(top_k, top_p, V);
    const FilterState st = filter_descend<FILTER_BINS0>(hist_cnt, hist_mass, FilterState{0ull, 0ull, 0u, 0u}, FILTER_SHIFT0,
                                                        lim.k, lim.P, dsc);
    if (threadIdx.x == 0) states[r] = st;
  }
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
filter_second_kernel(const float* __restrict__ logits, const float* __restrict__ temperatures,
                     const long long* __restrict__ top_ks, const float* __restrict__ top_ps, unsigned* hist_cnt,
                     unsigned long long* hist_mass, FilterState* __restrict__ states, const float2* __restrict__ norms,
                     unsigned* marks, float* __restrict__ list, int R, int V, int chunks) {
  pdl_prologue(logits, temperatures, top_ks, top_ps, norms);
  __shared__ unsigned s_cnt[FILTER_BINS1], s_low[FILTER_BINS1], s_high[FILTER_BINS1];
  __shared__ DescendScratch dsc;
  __shared__ float s_list[ARGMAX_CHUNK];
  __shared__ int s_listed;
  __shared__ bool s_last;
  const int r = blockIdx.y, c = blockIdx.x, lane = threadIdx.x & 31;
  const float temp = temperatures[r];
  const long long top_k = top_ks[r];
  const float top_p = top_ps[r];
  if (!row_is_filtered(temp, top_k, top_p)) return;
  const int lo = c * ARGMAX_CHUNK, hi = min(V, lo + ARGMAX_CHUNK);
  float x[PER_THREAD];
  load_chunk(logits + (size_t)r * V, lo, hi, x);
  FilterState st{__ldcg(&states[r].cnt_above), __ldcg(&states[r].mass_above), __ldcg(&states[r].prefix), 0u};
  const float2 norm = norms[r];
  for (int b = threadIdx.x; b < FILTER_BINS1; b += SAMPLE_THREADS) s_cnt[b] = s_low[b] = s_high[b] = 0u;
  if (threadIdx.x == 0) s_listed = 0;
  // the tokens that may have the prefix, side by side
  const Estimate est(temp, norm.x, norm.y);
  const float from = lower_bound(st.prefix, est), to = upper_bound(st.prefix | ((1u << FILTER_SHIFT0) - 1u), est);
  unsigned in[PER_THREAD];                   // the warp's, a bit a lane
  int found = 0;
#pragma unroll
  for (int j = 0; j < PER_THREAD; ++j) {
    const float y = est.log2p(x[j]);
    in[j] = __ballot_sync(0xffffffffu, lo + (int)threadIdx.x + j * SAMPLE_THREADS < hi && !(est.ok && (y < from || y > to)));
    found += __popc(in[j]);
  }
  __syncthreads();
  int at = 0;
  if (lane == 0 && found > 0) at = atomicAdd(&s_listed, found);
  at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
  for (int j = 0; j < PER_THREAD; ++j) {
    if ((in[j] >> lane) & 1u) s_list[at + __popc(in[j] & ((1u << lane) - 1u))] = x[j];
    at += __popc(in[j]);
  }
  __syncthreads();
  hist_cnt += (size_t)r * FILTER_BINS + FILTER_BINS0;
  hist_mass += (size_t)r * FILTER_BINS + FILTER_BINS0;
  const int n = s_listed;
  if (n > 0) {
    unsigned* listed = &marks[(size_t)r * ROW_MARKS + MARK_LISTED];
    for (int i = threadIdx.x; i - lane < n; i += SAMPLE_THREADS) {
      const float p = row_probability(i < n ? s_list[i] : 0.f, temp, norm.x, norm.y);
      const unsigned key = __float_as_uint(p);
      const bool mine = i < n && (key >> FILTER_SHIFT0) == (st.prefix >> FILTER_SHIFT0);
      count_token(p, (key >> FILTER_SHIFT1) & (FILTER_BINS1 - 1), mine, s_cnt, s_low, s_high);
      const unsigned ballot = __ballot_sync(0xffffffffu, mine);
      unsigned where = 0u;
      if (lane == 0 && ballot != 0u) where = atomicAdd(listed, (unsigned)__popc(ballot));
      where = __shfl_sync(0xffffffffu, where, 0) + __popc(ballot & ((1u << lane) - 1u));
      if (mine && where < (unsigned)FILTER_LIST) list[(size_t)r * FILTER_LIST + where] = p;
    }
    __syncthreads();
    add_histogram<FILTER_BINS1>(s_cnt, s_low, s_high, hist_cnt, hist_mass);
  }
  if (last_of_row(&marks[(size_t)r * ROW_MARKS + MARK_SECOND], chunks, &s_last)) {
    const FilterLimits lim(top_k, top_p, V);
    st = filter_descend<FILTER_BINS1>(hist_cnt, hist_mass, st, FILTER_SHIFT1, lim.k, lim.P, dsc);
    if (threadIdx.x == 0) states[R + r] = st;
    // a list that overflowed: the third pass counts into the first one's histogram
    if (__ldcg(&marks[(size_t)r * ROW_MARKS + MARK_LISTED]) > (unsigned)FILTER_LIST)
      for (int b = threadIdx.x; b < FILTER_BINS2; b += SAMPLE_THREADS) {
        hist_cnt[b - FILTER_BINS0] = 0u;
        hist_mass[b - FILTER_BINS0] = 0ull;
      }
  }
}

// The last 10 bits, from the listed probabilities that have the first 21: a row's first block; where the list is
// too short all of them, from the row.
__global__ void __launch_bounds__(SAMPLE_THREADS)
filter_third_kernel(const float* __restrict__ logits, const float* __restrict__ temperatures,
                    const long long* __restrict__ top_ks, const float* __restrict__ top_ps,
                    const FilterState* __restrict__ states, const float2* __restrict__ norms,
                    unsigned* marks, const float* __restrict__ list, unsigned* hist_cnt, unsigned long long* hist_mass,
                    unsigned* __restrict__ thresh, int R, int V) {
  pdl_prologue(logits, temperatures, top_ks, top_ps, states, norms, marks, list);
  __shared__ unsigned s_cnt[FILTER_BINS2];
  __shared__ unsigned long long s_mass[FILTER_BINS2];
  __shared__ DescendScratch dsc;
  __shared__ bool s_last;
  const int r = blockIdx.y, part = blockIdx.x, lane = threadIdx.x & 31;
  const float temp = temperatures[r];
  const long long top_k = top_ks[r];
  const float top_p = top_ps[r];
  if (!row_is_filtered(temp, top_k, top_p)) {
    if (part == 0 && threadIdx.x == 0) thresh[r] = 0u;
    return;
  }
  const FilterState st = states[R + r];
  const unsigned listed = __ldcg(&marks[(size_t)r * ROW_MARKS + MARK_LISTED]);
  const bool whole = listed <= (unsigned)FILTER_LIST;          // the list has them all
  if (whole && part > 0) return;
  const float2 norm = norms[r];
  for (int b = threadIdx.x; b < FILTER_BINS2; b += SAMPLE_THREADS) {
    s_cnt[b] = 0u;
    s_mass[b] = 0ull;
  }
  __syncthreads();
  const int n = whole ? (int)listed : V;
  const float* from = whole ? list + (size_t)r * FILTER_LIST : logits + (size_t)r * V;
  const int first = whole ? threadIdx.x : part * SAMPLE_THREADS + threadIdx.x;
  const int step = whole ? SAMPLE_THREADS : THIRD_BLOCKS * SAMPLE_THREADS;
#pragma unroll 4
  for (int i = first; i - lane < n; i += step) {
    float p = i < n ? from[i] : 0.f;
    if (!whole) p = row_probability(p, temp, norm.x, norm.y);
    const unsigned key = __float_as_uint(p);
    const bool mine = i < n && (key >> FILTER_SHIFT1) == (st.prefix >> FILTER_SHIFT1);
    const unsigned bin = key & (FILTER_BINS2 - 1);
    const unsigned long long m = (unsigned long long)(p * MASS_ONE);
    const unsigned bin0 = __shfl_sync(0xffffffffu, bin, 0);
    if (__all_sync(0xffffffffu, mine && bin == bin0)) {
      const unsigned long long sum = ((unsigned long long)__reduce_add_sync(0xffffffffu, (unsigned)(m >> 20)) << 20) +
                                     __reduce_add_sync(0xffffffffu, (unsigned)(m & 0xfffffull));
      if (lane == 0) {
        atomicAdd(&s_cnt[bin], 32u);
        atomicAdd(&s_mass[bin], sum);
      }
    } else if (mine) {
      atomicAdd(&s_cnt[bin], 1u);
      atomicAdd(&s_mass[bin], m);
    }
  }
  __syncthreads();
  const FilterLimits lim(top_k, top_p, V);
  FilterState last;
  if (whole) {
    last = filter_descend<FILTER_BINS2, true>(s_cnt, s_mass, st, 0, lim.k, lim.P, dsc);
  } else {
    hist_cnt += (size_t)r * FILTER_BINS;
    hist_mass += (size_t)r * FILTER_BINS;
    for (int b = threadIdx.x; b < FILTER_BINS2; b += SAMPLE_THREADS)
      if (s_cnt[b] != 0u) {
        atomicAdd(&hist_cnt[b], s_cnt[b]);
        atomicAdd(&hist_mass[b], s_mass[b]);
      }
    if (!last_of_row(&marks[(size_t)r * ROW_MARKS + MARK_THIRD], THIRD_BLOCKS, &s_last)) return;
    last = filter_descend<FILTER_BINS2>(hist_cnt, hist_mass, st, 0, lim.k, lim.P, dsc);
  }
  if (threadIdx.x == 0) thresh[r] = last.prefix;
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
gumbel_pick_kernel(const float* __restrict__ logits, const float* __restrict__ temperatures,
                   const long long* __restrict__ seeds, const long long* __restrict__ sample_pos,
                   const unsigned char* __restrict__ keep, const unsigned* __restrict__ thresh,
                   const float2* __restrict__ norms, const float* __restrict__ cmax, const float* __restrict__ csum,
                   float* __restrict__ pv, int* __restrict__ pi, int V, int chunks) {
  pdl_prologue(logits, temperatures, seeds, sample_pos, keep, thresh, norms, cmax, csum);
  __shared__ Best bscratch[32];
  __shared__ NormaliserScratch nsc;
  const int r = blockIdx.y, c = blockIdx.x;
  const float* row = logits + (size_t)r * V;
  const int lo = c * ARGMAX_CHUNK, hi = min(V, lo + ARGMAX_CHUNK);
  float x[PER_THREAD];
  load_chunk(row, lo, hi, x);
  const float temp = temperatures[r];
  const unsigned t = thresh != nullptr ? thresh[r] : 0u;       // of top-k / top-p
  Best b{-INFINITY, INT_MAX_};
  if (temp <= 0.f) {
#pragma unroll
    for (int j = 0; j < PER_THREAD; ++j) {
      const int i = lo + threadIdx.x + j * SAMPLE_THREADS;
      if (i < hi) b = better(b, Best{x[j], i});
    }
  } else {
    float mx, sum;
    if (norms != nullptr) {
      const float2 n = norms[r];
      mx = n.x;
      sum = n.y;
    } else {
      row_normaliser(cmax, csum, r, chunks, nsc, mx, sum);
    }
    const long long seed = seeds[r], pos = sample_pos[r];
    const unsigned char* krow = keep ? keep + (size_t)r * V : nullptr;
    const Estimate est(temp, mx, sum);
    const float from = lower_bound(t, est);
    // An upper bound of every id's score, in bits.  With v = 1 - u, exact, the noise is at most
    // -log(v), because -log(1 - v) >= v; log(p + 1e-10) is at most the larger of the two logarithms
    // plus what the smaller adds: 1e-10 / p below p = 2^-20, at most one bit beyond.
    float ub[PER_THREAD];
    unsigned alive = 0u;
    int top = -1;
    float top_ub = -INFINITY;
#pragma unroll
    for (int j = 0; j < PER_THREAD; ++j) {
      const int i = lo + threadIdx.x + j * SAMPLE_THREADS;
      const float y = est.log2p(x[j]);
      const unsigned long long step =
          ((unsigned long long)seed * 19349663ull) ^ ((unsigned long long)pos * 73856093ull);
      const unsigned hashed = (unsigned)((step * 8589934591ull) ^ ((unsigned long long)i * 479001599ull)) & 0xffffffu;
      const float v = (float)(0x1000000u - hashed) * (1.0f / 16777216.0f);
      ub[j] = fmaxf(y, -33.2192f) + (y > -20.f ? 2e-4f : 1.0f) - __log2f(v) + est.margin;
      if (!est.ok) ub[j] = INFINITY;
      if (i < hi && !(krow && !krow[i]) && !(est.ok && y < from)) {
        alive |= 1u << j;
        if (top < 0 || ub[j] > top_ub) {
          top = j;
          top_ub = ub[j];
        }
      }
    }
    // every thread's most promising id first, then whatever may still beat the best of those
    unsigned todo = top >= 0 ? 1u << top : 0u;
    alive &= ~todo;
#pragma unroll 1
    for (int round = 0; round < 2; ++round) {
      if (round == 1) {
        const float reached = block_best(b, bscratch).v * 1.4426950408889634f;
        const float slack = 1e-6f * fabsf(reached);
        todo = 0u;
#pragma unroll
        for (int j = 0; j < PER_THREAD; ++j)
          if (((alive >> j) & 1u) && !(ub[j] < reached - slack)) todo |= 1u << j;
      }
      while (todo != 0u) {
        const int i = lo + threadIdx.x + (__ffs(todo) - 1) * SAMPLE_THREADS;
        todo &= todo - 1u;
        const float p = row_probability(row[i], temp, mx, sum);
        if (__float_as_uint(p) < t) continue;
        b = better(b, Best{logf(p + 1e-10f) + seeded_gumbel(seed, pos, i), i});
      }
    }
  }
  b = block_best(b, bscratch);
  if (threadIdx.x == 0) {
    pv[(size_t)r * chunks + c] = b.v;
    pi[(size_t)r * chunks + c] = b.i;
  }
}

}  // namespace

extern "C" {

int dib_argmax(const float* logits, int* out, int R, int V, cudaStream_t st) {
  if (R == 0) return DIB_OK;
  if (V < 1) return DIB_BAD_SIZE;
  dib_launch(argmax_kernel, dim3(R), dim3(1024), 0, st, logits, out, V);
  DIB_CHECK_LAUNCH();
  return DIB_OK;
}

int dib_argmax_chunks(int V) { return (V + ARGMAX_CHUNK - 1) / ARGMAX_CHUNK; }

// scratch_v / scratch_i: [R, dib_argmax_chunks(V)]
int dib_argmax_two_stage(const float* logits, float* scratch_v, int* scratch_i, int* out, int R,
                         int V, cudaStream_t st) {
  if (R == 0) return DIB_OK;
  if (V < 1 || R > 65535) return DIB_BAD_SIZE;
  const int chunks = (V + ARGMAX_CHUNK - 1) / ARGMAX_CHUNK;
  dib_launch(argmax_partial_kernel, dim3(dim3(chunks, R)), dim3(256), 0, st, logits, scratch_v, scratch_i, V, chunks);
  DIB_CHECK_LAUNCH();
  dib_launch(argmax_final_kernel, dim3(R), dim3(64), 0, st, scratch_v, scratch_i, out, chunks);
  DIB_CHECK_LAUNCH();
  return DIB_OK;
}

int dib_gumbel_sample(const float* logits, const float* temperatures, const long long* seeds,
                      const long long* sample_pos, const unsigned char* keep, int* out, int R,
                      int V, cudaStream_t st) {
  if (R == 0) return DIB_OK;
  if (V < 1) return DIB_BAD_SIZE;
  dib_launch(gumbel_sample_kernel, dim3(R), dim3(1024), 0, st, logits, temperatures, seeds, sample_pos, keep, out, V);
  DIB_CHECK_LAUNCH();
  return DIB_OK;
}

// The same in chunks (see gumbel_stats_kernel).  scratch_f: float [3, R, chunks];
// scratch_i: int [R, chunks], chunks = dib_argmax_chunks(V).
// top_ks / top_ps (both or neither): per-row top-k (<= 0: off) and top-p (>= 1: off),
// applied by a threshold found without a sort.  thresh: unsigned [R], receives the bits of
// each row's smallest kept probability (0 = all kept); hist: scratch of dib_filter_scratch(R)
// bytes, 8-byte aligned (more than FILTER_ROWS rows go through it in turn, in stream order).
long long dib_filter_scratch(int R) {
  return (R < FILTER_ROWS ? R : FILTER_ROWS) *
         (FILTER_BINS * 12ll + 2 * (long long)sizeof(FilterState) + (long long)sizeof(float2) + 4ll * ROW_MARKS +
          4ll * FILTER_LIST);
}

int dib_gumbel_sample_chunked(const float* logits, const float* temperatures, const long long* seeds,
                              const long long* sample_pos, const unsigned char* keep,
                              const long long* top_ks, const float* top_ps, unsigned* thresh,
                              void* hist, float* scratch_f, int* scratch_i, int* out, int R, int V,
                              cudaStream_t st) {
  if (R == 0) return DIB_OK;
  if (V < 1 || R > 65535) return DIB_BAD_SIZE;
  const int chunks = (V + ARGMAX_CHUNK - 1) / ARGMAX_CHUNK;
  const bool filtered = top_ks != nullptr && top_ps != nullptr && thresh != nullptr && hist != nullptr;
  if (filtered && reinterpret_cast<uintptr_t>(hist) % 8 != 0) return DIB_BAD_ALIGN;
  if (filtered && R > FILTER_ROWS) {       // rows in turn through the same scratch (it is 100 KB a row)
    for (int r = 0; r < R; r += FILTER_ROWS) {
      const int n = R - r < FILTER_ROWS ? R - r : FILTER_ROWS;
      const int status = dib_gumbel_sample_chunked(
          logits + (size_t)r * V, temperatures + r, seeds + r, sample_pos + r, keep != nullptr ? keep + (size_t)r * V : keep,
          top_ks + r, top_ps + r, thresh + r, hist, scratch_f, scratch_i, out + r, n, V, st);
      if (status != DIB_OK) return status;
    }
    return DIB_OK;
  }
  float* cmax = scratch_f;
  float* csum = scratch_f + (size_t)R * chunks;
  float* pv = scratch_f + 2 * (size_t)R * chunks;
  // masses, the rows' states and normalisers, then what needs 4 bytes only
  unsigned long long* hist_mass = filtered ? reinterpret_cast<unsigned long long*>(hist) : nullptr;
  FilterState* states = filtered ? reinterpret_cast<FilterState*>(hist_mass + (size_t)R * FILTER_BINS) : nullptr;
  float2* norms = filtered ? reinterpret_cast<float2*>(states + (size_t)2 * R) : nullptr;
  unsigned* hist_cnt = filtered ? reinterpret_cast<unsigned*>(norms + R) : nullptr;
  unsigned* marks = filtered ? hist_cnt + (size_t)R * FILTER_BINS : nullptr;
  float* list = filtered ? reinterpret_cast<float*>(marks + (size_t)R * ROW_MARKS) : nullptr;
  const dim3 grid(chunks, R), block(SAMPLE_THREADS);
  dib_launch(gumbel_stats_kernel, grid, block, 0, st, logits, temperatures, cmax, csum, hist_cnt, hist_mass, marks, V,
             chunks);
  DIB_CHECK_LAUNCH();
  if (filtered) {
    dib_launch(filter_first_kernel, grid, block, 0, st, logits, temperatures, top_ks, top_ps, (const float*)cmax,
               (const float*)csum, hist_cnt, hist_mass, states, norms, marks, V, chunks);
    DIB_CHECK_LAUNCH();
    dib_launch(filter_second_kernel, grid, block, 0, st, logits, temperatures, top_ks, top_ps, hist_cnt, hist_mass,
               states, (const float2*)norms, marks, list, R, V, chunks);
    DIB_CHECK_LAUNCH();
    dib_launch(filter_third_kernel, dim3(THIRD_BLOCKS, R), block, 0, st, logits, temperatures, top_ks, top_ps,
               (const FilterState*)states, (const float2*)norms, marks, (const float*)list, hist_cnt, hist_mass, thresh, R,
               V);
    DIB_CHECK_LAUNCH();
  }
  dib_launch(gumbel_pick_kernel, grid, block, 0, st, logits, temperatures, seeds, sample_pos, keep,
             filtered ? (const unsigned*)thresh : (const unsigned*)nullptr, (const float2*)norms, (const float*)cmax,
             (const float*)csum, pv, scratch_i, V, chunks);
  DIB_CHECK_LAUNCH();
  dib_launch(argmax_final_kernel, dim3(R), dim3(64), 0, st, (const float*)pv, (const int*)scratch_i, out,
             chunks);
  DIB_CHECK_LAUNCH();
  return DIB_OK;
}

}  // extern "C"

// Exact temperature / top-k / top-p / categorical selection over the WHOLE vocabulary, a cluster of CTAs per row, plus the
// sequence bookkeeping of the step — the second (and last) launch of a sampling decode step at any tp.
//
// Reference behaviour: the HF Flax warpers as configured by jax_llama/generation.py:28-41 —
// logits / T → top-k (if set) → top-p with min_tokens_to_keep = 1 (sorted descending, a token is kept while the
// probability mass before it is < top_p) → categorical; temperature 0 = arg-max.  A first form ran this on at most 64
// candidates per row, so `top_k=None` silently meant "nucleus over the 64 most likely tokens" on the GPU and a
// plateau of equal logits could overflow the candidate list.  This kernel has no candidate budget:
//
//   * every token gets the 64-bit sort key (order-preserving bits of its scaled logit, ~index): larger key = better,
//     equal logits order by LOWER index — selection is deterministic whatever the thread arrival order;
//   * the question asked of a row is always "the element whose interval of the descending cumulative sum contains `target`":
//     with unit weights it is the k-th largest element (top-k), with probability weights the nucleus boundary (top-p) and the
//     sampled token (inverse CDF at u·Z).  Probabilities are exp(z − max) in 2^-40 fixed point, so every sum is an integer sum:
//     associative, hence bit-identical on every rank and every run (float atomics are not);
//   * a cluster of up to 8 CTAs shares a row.  ONE pass over the logits fills a histogram (counts and masses) over equal steps of
//     z below the row's maximum; its prefix sums answer all three questions down to a bin, because top-k and top-p only cut the
//     same cumulative sum off at an earlier point.  The few elements of all their bins are then gathered and ranked exactly; a bin with
//     more than SF_CAND elements (plateaus, coarse logits) is first narrowed by histograms over its own (key, ~index) range.
//     What bounds it is the chain of cluster barriers and short passes, not the 0.5 MB of a row: 4 rows of 128256, top-p 0.95, on
//     one B200: 632 us with one CTA per row and three radix passes per question (the top bits of normal logits fall into a few
//     dozen bins, so its 64-bit shared-memory atomics serialised), 29 us with one gather per question, 23 us with one gather for all;
//   * rows that hold a NaN or whose maximum is not finite take the radix select that the first form of this kernel ran for every
//     row (sf_select): their masses are not sums of probabilities, and what they return stays what it was.
//   * tensor parallelism: the decode kernel stores every rank's logits shard into every rank's [B, V] buffer with
//     multimem.st, so all ranks run this kernel on identical inputs with the same Philox stream (seed, step, row) and
//     pick the same token without a broadcast.  The kernel first waits for the arg-max candidate packets of all ranks
//     (they are published after a system fence that follows the logits stores).
#include <cooperative_groups.h>

#include "common.cuh"
#include "jllama_b200.h"

namespace cg = cooperative_groups;

namespace jl {

constexpr int SF_THREADS = 1024;
constexpr int SF_BINS = 2048;
constexpr int SF_CAND = 256;                       // elements ranked directly (four threads each)
constexpr int SF_MAX_CLUSTER = 8;
constexpr float SF_STEP = 2047.0f / 28.0f;         // bins per unit of z: beyond 28 below the maximum a mass is zero (28 > 40 ln 2)
constexpr float SF_FIX = 1099511627776.f;          // 2^40

__device__ __forceinline__ uint32_t sf_key(float z) {
  if (!(z == z)) return 0u;                          // NaN sorts last
  const uint32_t u = __float_as_uint(z);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// same generator as sampling.cu (Philox-4x32-10 keyed by seed, counter = (step, row))
__device__ __forceinline__ float sf_uniform(unsigned long long seed, unsigned int step, unsigned int row) {
  unsigned int c0 = step, c1 = row, c2 = 0x9E3779B9u, c3 = 0xBB67AE85u;
  unsigned int k0 = (unsigned int)seed, k1 = (unsigned int)(seed >> 32);
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const unsigned int hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
    const unsigned int hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
    const unsigned int n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
    c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
  }
  return ((c0 >> 8) + 0.5f) * (1.0f / 16777216.0f);      // (0, 1)
}

struct SfRow {
  const float* x;           // logits of this row
  int V;
  float inv_temp, zmax;     // z = x · inv_temp; zmax = max z
  // current kept set: elements with key > kmin, or key == kmin and index <= imax (lower index = better)
  uint32_t kmin;
  int imax;
};

__device__ __forceinline__ bool sf_in_set(const SfRow& r, uint32_t key, int i) {
  return key > r.kmin || (key == r.kmin && i <= r.imax);
}
// z = x · inv_temp rounded to fp32, and its distance to the maximum likewise: never contracted into one operation, so that every pass
// over a row sees the same keys, bins and masses
__device__ __forceinline__ float sf_scaled(float x, float inv_temp) { return __fmul_rn(x, inv_temp); }
__device__ __forceinline__ unsigned long long sf_mass(const SfRow& r, float z) {
  return (unsigned long long)(exp2f(__fmul_rn(__fsub_rn(z, r.zmax), 1.4426950408889634f)) * SF_FIX);
}

// Descending scan of the histogram (warp 0): the bin in which the running sum (starting at `base`) first exceeds
// `target`, and the sum before that bin.  A target at or beyond the total (rounding of a fraction) selects the last
// non-empty bin.
__device__ void sf_scan(const unsigned long long* hist, int nbins, unsigned long long target, unsigned long long base,
                        int* out_bin, unsigned long long* out_before, unsigned long long* out_total) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  const int per = nbins / 32;                            // lane 0 owns the highest bins
  unsigned long long s = 0;
  for (int j = 0; j < per; ++j) s += hist[nbins - 1 - (lane * per + j)];
  unsigned long long incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const unsigned long long total = __shfl_sync(0xffffffffu, incl, 31) + base;
  const unsigned long long excl = incl - s + base;
  const unsigned cross = __ballot_sync(0xffffffffu, s > 0 && target < excl + s);
  const unsigned nonempty = __ballot_sync(0xffffffffu, s > 0);
  int owner;
  bool past_end = false;
  if (cross) owner = __ffs(cross) - 1;
  else { owner = nonempty ? 31 - __clz(nonempty) : 0; past_end = true; }
  if (lane == owner) {
    unsigned long long acc = excl, before = excl;
    int bin = nbins - 1 - lane * per;
    for (int j = 0; j < per; ++j) {
      const int b = nbins - 1 - (lane * per + j);
      const unsigned long long h = hist[b];
      if (h > 0) { bin = b; before = acc; if (!past_end && acc + h > target) break; }
      acc += h;
    }
    *out_bin = bin; *out_before = before;
  }
  if (lane == 0) *out_total = total;
}

// The element of the kept set whose interval [before, before + w) of the descending cumulative sum contains `target`
// (w = 1 per element if BY_COUNT, else its fixed-point probability).  Returns (key, index); *before_out = sum strictly
// before that element, *set_total = sum over the whole kept set (valid after the first level).
template <bool BY_COUNT>
__device__ void sf_select(const SfRow& r, unsigned long long target, bool target_is_fraction, double fraction,
                          unsigned long long* hist, int* s_bin, unsigned long long* s_before, unsigned long long* s_total,
                          int* s_idx, uint32_t* key_out, int* idx_out, unsigned long long* before_out,
                          unsigned long long* total_out) {
  uint32_t prefix = 0;            // key bits fixed so far (top `done` bits)
  int done = 0;
  unsigned long long before = 0, set_total = 0;
  const int widths[3] = {11, 11, 10};
#pragma unroll 1
  for (int level = 0; level < 3; ++level) {
    const int w = widths[level], shift = 32 - done - w, nb = 1 << w;
    for (int b = threadIdx.x; b < SF_BINS; b += SF_THREADS) hist[b] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < r.V; i += SF_THREADS) {
      const float z = sf_scaled(r.x[i], r.inv_temp);
      const uint32_t key = sf_key(z);
      if (!sf_in_set(r, key, i)) continue;
      if (done > 0 && (key >> (32 - done)) != (prefix >> (32 - done))) continue;
      const int bin = (key >> shift) & (nb - 1);
      atomicAdd(&hist[bin], BY_COUNT ? 1ull : sf_mass(r, z));
    }
    __syncthreads();
    if (level == 0 && target_is_fraction) {
      // the target is a fraction of the kept set's total, known only now: target = max(fraction·Z, 1) − 1
      // (a token is kept while the mass before it is < fraction·Z)
      if (threadIdx.x < 32) {
        unsigned long long s = 0;
        for (int b = threadIdx.x; b < nb; b += 32) s += hist[b];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) {
          unsigned long long t = (unsigned long long)((double)s * fraction);
          if (t > s) t = s;
          *s_total = t > 0 ? t - 1 : 0;
        }
      }
      __syncthreads();
      target = *s_total;
      __syncthreads();
    }
    sf_scan(hist, nb, target, before, s_bin, s_before, s_total);
    __syncthreads();
    prefix |= (uint32_t)(*s_bin) << shift;
    before = *s_before;
    if (level == 0) set_total = *s_total;
    done += w;
    __syncthreads();
  }
  // exact ties: elements of the set with key == prefix all weigh the same; the r-th lowest index crosses
  unsigned long long wt = 1;
  if (!BY_COUNT) {
    // weight of one tied element: recompute from the key (z is not recoverable bit-exactly from the key only for NaN)
    const uint32_t u = (prefix & 0x80000000u) ? (prefix & 0x7fffffffu) : ~prefix;
    wt = sf_mass(r, __uint_as_float(u));
  }
  unsigned long long rank = wt > 0 ? (target >= before ? (target - before) / wt : 0) : 0;      // 0-based among ties
  // count ties and find the (rank)-th lowest index: lowest index by atomicMin when rank == 0 (the common case)
  if (threadIdx.x == 0) { *s_idx = 0x7fffffff; *s_bin = 0; }
  __syncthreads();
  for (int i = threadIdx.x; i < r.V; i += SF_THREADS) {
    const uint32_t key = sf_key(sf_scaled(r.x[i], r.inv_temp));
    if (key == prefix && sf_in_set(r, key, i)) { atomicMin(s_idx, i); atomicAdd(s_bin, 1); }
  }
  __syncthreads();
  int idx = *s_idx;
  const int n_ties = *s_bin;
  __syncthreads();
  if (rank >= (unsigned long long)n_ties) rank = n_ties > 0 ? n_ties - 1 : 0;
  if (rank > 0) {
    // radix select over the index (17 bits: 9 + 8) among the ties, ascending
    int ipre = 0, idone = 0;
    unsigned long long ibefore = 0;
    const int iw[2] = {9, 8};
#pragma unroll 1
    for (int level = 0; level < 2; ++level) {
      const int w = iw[level], shift = 17 - idone - w, nb = 1 << w;
      for (int b = threadIdx.x; b < SF_BINS; b += SF_THREADS) hist[b] = 0;
      __syncthreads();
      for (int i = threadIdx.x; i < r.V; i += SF_THREADS) {
        const uint32_t key = sf_key(sf_scaled(r.x[i], r.inv_temp));
        if (key != prefix || !sf_in_set(r, key, i)) continue;
        if (idone > 0 && (i >> (17 - idone)) != (ipre >> (17 - idone))) continue;
        // ascending index order = descending (nb − 1 − digit)
        atomicAdd(&hist[nb - 1 - ((i >> shift) & (nb - 1))], 1ull);
      }
      __syncthreads();
      sf_scan(hist, nb, rank, ibefore, s_bin, s_before, s_total);
      __syncthreads();
      ipre |= (nb - 1 - *s_bin) << shift;
      ibefore = *s_before;
      idone += w;
      __syncthreads();
    }
    idx = ipre;
  }
  *key_out = prefix; *idx_out = idx;
  *before_out = before + rank * wt;
  *total_out = set_total;
}

struct SampleFullParams {
  const float* logits;      // [B, ld] fp32 (full vocabulary)
  int V, ld, B;
  float inv_temp, top_p;
  int top_k;
  unsigned long long seed;
  const int* step;
  int* tok;
  // wait for the other ranks' logits shards (tp > 1): candidate packets of the decode kernel, see decode_mega.cu
  const uint2* cand; const unsigned int* gen; int tp, grid, two_l, rank;
  // bookkeeping (advance_kernel), done by the last CTA to finish
  int* ticket; int* next_ids; int* finished; int* sequences; int max_len, eos, pad;
  int* cur_len; int* cache_len; int* step_rw; int* n_unfinished;
};

// Rows whose masses are not probabilities (a NaN, an infinite maximum): one CTA, radix selects over the whole row.
__device__ int sf_radix_row(SfRow r, int top_k, float top_p, float u01, unsigned long long* hist) {
  __shared__ unsigned long long s_before, s_total;
  __shared__ int s_bin, s_idx;
  uint32_t key; int idx; unsigned long long before, total;
  if (top_k > 0 && top_k < r.V) {
    sf_select<true>(r, (unsigned long long)(top_k - 1), false, 0.0, hist, &s_bin, &s_before, &s_total, &s_idx, &key, &idx, &before, &total);
    r.kmin = key; r.imax = idx;
  }
  if (top_p < 1.0f) {
    sf_select<false>(r, 0, true, (double)top_p, hist, &s_bin, &s_before, &s_total, &s_idx, &key, &idx, &before, &total);
    r.kmin = key; r.imax = idx;
  }
  // inverse CDF over the kept set, descending order
  sf_select<false>(r, 0, true, (double)u01, hist, &s_bin, &s_before, &s_total, &s_idx, &key, &idx, &before, &total);
  return idx;
}

struct SfShared {
  // this CTA's histogram of the level in work: counts, and masses (< 2^41) in three 14-bit digits, so that 32-bit atomics cannot
  // overflow for a slice of up to 2^17 elements
  unsigned int cnt[SF_BINS], m0[SF_BINS], m1[SF_BINS], m2[SF_BINS];
  // rank 0 of the cluster: prefix sums before each bin (one more entry: the total) of the first level, and of the narrowing level
  unsigned long long pm[SF_BINS + 1], rm[SF_BINS + 1];
  unsigned int pc[SF_BINS + 1], rc[SF_BINS + 1];
  unsigned long long cand[SF_CAND], cmass[SF_CAND];
  unsigned long long warp_m[32];
  unsigned int warp_c[32];
  // rank 0's decisions, written into every CTA
  int bin, n;
  unsigned long long klo, khi;
  // rank 0: where the gathered elements and the range of a bin meet; the answer of a question
  unsigned int n_cand;
  unsigned long long rlo[SF_MAX_CLUSTER], rhi[SF_MAX_CLUSTER];
  unsigned long long base_m; unsigned int base_c;
  unsigned long long res_comp, res_before, res_mass;
  // all questions at once: ranges of bins to gather (rank 0's decision, written into every CTA), per candidate its bin and the sums before it
  int ranges, range_lo[3], range_hi[3], at[2];
  int cbin[SF_CAND];
  unsigned long long cbefore[SF_CAND];
  unsigned int crank_of[SF_CAND];
};

struct SfBest {
  unsigned long long best[SF_MAX_CLUSTER];         // per CTA: best (key, ~index) of its slice
  unsigned int odd[SF_MAX_CLUSTER];                // per CTA: it saw a NaN
  unsigned long long best_local;
  unsigned int odd_local;
};

// (a barrier of one CTA costs less than a cluster's)
__device__ __forceinline__ void sf_sync(cg::cluster_group& cl, int size) {
  if (size > 1) cl.sync(); else __syncthreads();
}

// "I have started" without an order of memory: the barrier's wait comes after the pass over the slice, which hides it
__device__ __forceinline__ void sf_cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void sf_cluster_wait() { asm volatile("barrier.cluster.wait;" ::: "memory"); }

// One row as its cluster sees it.
struct SfCluster {
  SfShared* s;
  const float* x;
  int V, lo, hi, vec;           // this CTA's slice [lo, hi)
  float inv_temp, zmax;
  uint32_t kmax;                // key of the row's maximum
  int rank, size;
  bool count_all;               // elements without mass count too (a top-k question will be asked)
  SfRow row;

  template <int N = 4, typename F> __device__ __forceinline__ void for_slice(F f) const {
    if (vec) {                                              // lo is a multiple of four
      // N loads in flight: a slice of a 128 k row is four rounds, each a memory latency when they follow one another (two for the arg-max
      // alone, whose two CTAs per SM have 32 registers a thread: 64 rows of 128256 24 -> 18 us)
      for (int i0 = lo + 4 * (int)threadIdx.x; i0 < hi; i0 += 4 * N * SF_THREADS) {
        float4 v[N];
#pragma unroll
        for (int u = 0; u < N; ++u)
          if (i0 + 4 * SF_THREADS * u + 4 <= hi) v[u] = *reinterpret_cast<const float4*>(x + i0 + 4 * SF_THREADS * u);
#pragma unroll
        for (int u = 0; u < N; ++u) {
          const int i = i0 + 4 * SF_THREADS * u;
          if (i + 4 <= hi) {
            f(v[u].x, i); f(v[u].y, i + 1); f(v[u].z, i + 2); f(v[u].w, i + 3);
          } else {
            for (int j = i; j < hi; ++j) f(x[j], j);
          }
        }
      }
    } else {
      for (int i = lo + (int)threadIdx.x; i < hi; i += SF_THREADS) f(x[i], i);
    }
  }
  // monotone in z: larger z, smaller or equal bin
  __device__ __forceinline__ int bin_of(float z) const {
    const float d = __fmul_rn(__fsub_rn(zmax, z), SF_STEP);
    return d < (float)(SF_BINS - 1) ? (int)d : SF_BINS - 1;
  }
  static __device__ __forceinline__ unsigned long long comp(uint32_t key, int i) {
    return ((unsigned long long)key << 32) | (unsigned)(0x7fffffff - i);
  }
  static __device__ __forceinline__ float z_of(unsigned long long c) {
    const uint32_t k = (uint32_t)(c >> 32);
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
  }
  __device__ __forceinline__ void add(int bin, unsigned long long m) const {
    atomicAdd(&s->cnt[bin], 1u);
    if (m) {
      const unsigned d0 = (unsigned)m & 0x3fffu, d1 = (unsigned)(m >> 14) & 0x3fffu, d2 = (unsigned)(m >> 28);
      if (d0) atomicAdd(&s->m0[bin], d0);
      if (d1) atomicAdd(&s->m1[bin], d1);
      if (d2) atomicAdd(&s->m2[bin], d2);
    }
  }
  __device__ __forceinline__ void clear() const {
    for (int b = threadIdx.x; b < SF_BINS; b += SF_THREADS) { s->cnt[b] = 0; s->m0[b] = 0; s->m1[b] = 0; s->m2[b] = 0; }
    __syncthreads();
  }
  // all CTAs' histograms -> exclusive prefix sums in rank 0 (pm / pc, or rm / rc); every CTA adds up its share of the bins
  __device__ void merge(bool narrow) const {
    cg::cluster_group cl = cg::this_cluster();
    sf_sync(cl, size);                                              // every CTA's histogram is complete
    SfShared* lead = cl.map_shared_rank(s, 0);
    unsigned long long* tm = narrow ? lead->rm : lead->pm;
    unsigned int* tc = narrow ? lead->rc : lead->pc;
    const int share = SF_BINS / size;
    for (int b = rank * share + threadIdx.x; b < (rank + 1) * share; b += SF_THREADS) {
      unsigned long long m = 0;
      unsigned int c = 0;
#pragma unroll
      for (int r = 0; r < SF_MAX_CLUSTER; ++r) {                    // (unrolled: all CTAs' numbers on their way at once)
        if (r >= size) continue;
        const SfShared* o = cl.map_shared_rank(s, r);
        c += o->cnt[b];
        m += (unsigned long long)o->m0[b] + ((unsigned long long)o->m1[b] << 14) + ((unsigned long long)o->m2[b] << 28);
      }
      tm[b] = m; tc[b] = c;
    }
    sf_sync(cl, size);                                              // rank 0 holds all totals
    if (rank != 0) return;
    unsigned long long* lm = narrow ? s->rm : s->pm;
    unsigned int* lc = narrow ? s->rc : s->pc;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const unsigned long long m0 = lm[2 * t], m1 = lm[2 * t + 1];
    const unsigned int c0 = lc[2 * t], c1 = lc[2 * t + 1];
    unsigned long long im = m0 + m1;
    unsigned int ic = c0 + c1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long a = __shfl_up_sync(0xffffffffu, im, o);
      const unsigned int c = __shfl_up_sync(0xffffffffu, ic, o);
      if (lane >= o) { im += a; ic += c; }
    }
    if (lane == 31) { s->warp_m[w] = im; s->warp_c[w] = ic; }
    __syncthreads();
    if (w == 0) {
      unsigned long long a = s->warp_m[lane];
      unsigned int c = s->warp_c[lane];
      const unsigned long long a0 = a;
      const unsigned int cc0 = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_up_sync(0xffffffffu, a, o);
        const unsigned int v = __shfl_up_sync(0xffffffffu, c, o);
        if (lane >= o) { a += u; c += v; }
      }
      s->warp_m[lane] = a - a0; s->warp_c[lane] = c - cc0;
    }
    __syncthreads();
    const unsigned long long em = s->warp_m[w] + im - (m0 + m1);
    const unsigned int ec = s->warp_c[w] + ic - (c0 + c1);
    lm[2 * t] = em; lm[2 * t + 1] = em + m0;
    lc[2 * t] = ec; lc[2 * t + 1] = ec + c0;
    if (t == SF_THREADS - 1) { lm[SF_BINS] = em + m0 + m1; lc[SF_BINS] = ec + c0 + c1; }
    __syncthreads();
  }
  // rank 0: the bin whose interval holds `target` (relative to the prefix arrays) -> s->bin, s->n, base_m / base_c advanced
  __device__ __forceinline__ void find(const unsigned long long* lm, const unsigned int* lc, bool by_count, unsigned long long target) const {
    if (threadIdx.x == 0) { s->bin = SF_BINS - 1; s->n = 0; }      // (a target beyond the total: nothing)
    __syncthreads();
    for (int b = threadIdx.x; b < SF_BINS; b += SF_THREADS) {
      const unsigned long long a = by_count ? lc[b] : lm[b], e = by_count ? lc[b + 1] : lm[b + 1];
      if (a <= target && target < e) { s->bin = b; s->n = (int)(lc[b + 1] - lc[b]); }
    }
    __syncthreads();
  }
  // rank 0's bin, n and range into every CTA
  __device__ __forceinline__ void publish() const {
    cg::cluster_group cl = cg::this_cluster();
    if (rank == 0) {
      __syncthreads();
      if (threadIdx.x > 0 && (int)threadIdx.x < size) {
        SfShared* o = cl.map_shared_rank(s, (int)threadIdx.x);
        o->bin = s->bin; o->n = s->n; o->klo = s->klo; o->khi = s->khi;
      }
    }
    sf_sync(cl, size);
  }
  // The element whose interval of the descending cumulative sum (counts or masses) holds `target` (rank 0's value counts; it lies
  // below the total).  Executed by all CTAs of the cluster in step; the answer is in rank 0's res_*.
  __device__ void select(bool by_count, unsigned long long target) const {
    cg::cluster_group cl = cg::this_cluster();
    SfShared* lead = cl.map_shared_rank(s, 0);
    if (rank == 0) {
      find(s->pm, s->pc, by_count, target);
      if (threadIdx.x == 0) {
        s->base_m = s->pm[s->bin]; s->base_c = s->pc[s->bin];
        s->n_cand = 0;
        s->res_comp = 0x7fffffffull; s->res_before = 0; s->res_mass = 0;
      }
    }
    publish();
    int bin = s->bin, n = s->n;
    unsigned long long klo = 0, khi = ~0ull;
    if (n > SF_CAND) {                                      // too many to rank: the range of the bin's elements ...
      unsigned long long mn = ~0ull, mx = 0ull;
      for_slice([&](float v, int i) {
        const float z = sf_scaled(v, inv_temp);
        if (bin_of(z) != bin || !(count_all || sf_mass(row, z) > 0)) return;
        const unsigned long long c = comp(sf_key(z), i);
        mn = c < mn ? c : mn;
        mx = c > mx ? c : mx;
      });
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long a = __shfl_xor_sync(0xffffffffu, mn, o), b = __shfl_xor_sync(0xffffffffu, mx, o);
        mn = a < mn ? a : mn;
        mx = b > mx ? b : mx;
      }
      if ((threadIdx.x & 31) == 0) { s->warp_m[threadIdx.x >> 5] = mn; s->cmass[threadIdx.x >> 5] = mx; }
      __syncthreads();
      if (threadIdx.x == 0) {
        for (int w = 1; w < SF_THREADS / 32; ++w) {
          mn = s->warp_m[w] < mn ? s->warp_m[w] : mn;
          mx = s->cmass[w] > mx ? s->cmass[w] : mx;
        }
        lead->rlo[rank] = mn; lead->rhi[rank] = mx;
      }
      sf_sync(cl, size);
      if (rank == 0 && threadIdx.x == 0) {
        for (int r = 0; r < size; ++r) {
          mn = s->rlo[r] < mn ? s->rlo[r] : mn;
          mx = s->rhi[r] > mx ? s->rhi[r] : mx;
        }
        s->klo = mn; s->khi = mx;
      }
      publish();
      klo = s->klo; khi = s->khi;
      for (int level = 0; level < 6 && n > SF_CAND; ++level) {       // ... cut into 2048 parts, until few enough are left (64 bits: six times)
        const unsigned long long range = khi - klo;
        const int bits = 64 - __clzll((long long)range), shift = bits > 11 ? bits - 11 : 0;
        clear();
        for_slice([&](float v, int i) {
          const float z = sf_scaled(v, inv_temp);
          const unsigned long long c = comp(sf_key(z), i);
          if (c < klo || c > khi) return;
          const unsigned long long m = sf_mass(row, z);
          if (!count_all && m == 0) return;
          add((int)((khi - c) >> shift), m);
        });
        merge(true);
        if (rank == 0) {
          find(s->rm, s->rc, by_count, target - (by_count ? (unsigned long long)s->base_c : s->base_m));
          if (threadIdx.x == 0) {
            s->base_m += s->rm[s->bin]; s->base_c += s->rc[s->bin];
            const unsigned long long top = khi - ((unsigned long long)s->bin << shift);
            const unsigned long long span = (1ull << shift) - 1ull;
            s->khi = top;
            s->klo = top - klo > span ? top - span : klo;
          }
        }
        publish();
        n = s->n; klo = s->klo; khi = s->khi;
      }
      bin = -1;
    }
    for_slice([&](float v, int i) {                          // gather
      const float z = sf_scaled(v, inv_temp);
      if (bin >= 0 && bin_of(z) != bin) return;
      const unsigned long long c = comp(sf_key(z), i);
      if (bin < 0 && (c < klo || c > khi)) return;
      if (!count_all && sf_mass(row, z) == 0) return;
      const unsigned slot = atomicAdd(&lead->n_cand, 1u);
      if (slot < SF_CAND) lead->cand[slot] = c;
    });
    sf_sync(cl, size);
    if (rank != 0) return;
    const int nc = min((int)s->n_cand, SF_CAND);
    if ((int)threadIdx.x < nc) s->cmass[threadIdx.x] = sf_mass(row, z_of(s->cand[threadIdx.x]));
    __syncthreads();
    const int c = threadIdx.x >> 2;
    const unsigned long long mine = c < nc ? s->cand[c] : 0ull;
    unsigned long long bm = 0;
    unsigned int bc = 0;
    for (int j = threadIdx.x & 3; j < nc; j += 4)
      if (s->cand[j] > mine) { bm += s->cmass[j]; ++bc; }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) { bm += __shfl_xor_sync(0xffffffffu, bm, o); bc += __shfl_xor_sync(0xffffffffu, bc, o); }
    if (c < nc && (threadIdx.x & 3) == 0) {
      bm += s->base_m;
      const unsigned long long m = s->cmass[c];
      const bool hit = by_count ? (unsigned long long)bc + s->base_c == target : bm <= target && target - bm < m;
      if (hit) { s->res_comp = mine; s->res_before = bm; s->res_mass = m; }
    }
    __syncthreads();
  }

  // rank 0: the bins that hold lo and hi (masses, below the total) -> s->at
  __device__ __forceinline__ void find_two(unsigned long long lo_t, unsigned long long hi_t) const {
    for (int b = threadIdx.x; b < SF_BINS; b += SF_THREADS) {
      const unsigned long long a = s->pm[b], e = s->pm[b + 1];
      if (a <= lo_t && lo_t < e) s->at[0] = b;
      if (a <= hi_t && hi_t < e) s->at[1] = b;
    }
    __syncthreads();
  }
  // Every question of the row from one gather.  What top-k keeps lies between the sums before and behind the bin of its boundary, so the
  // next target lies in a range of bins, almost always one, and so on: the bins of all answers are known before any answer is, and when they
  // hold few enough elements these are gathered together and the questions answered one after the other by rank 0 alone.  The sums are the
  // same integers that select() forms.  False (in every CTA): more than SF_CAND elements, nothing was answered, select() goes on.
  // It saves a pass over the slice and two cluster barriers per question: 4 rows of 128256, top-k 50 and top-p 0.9, 36 -> 27 us from one
  // event to the next; top-p 0.95 alone 32 -> 27; 200 rows, both, 222 -> 135.
  template <typename Target>
  __device__ bool all_at_once(int top_k, float top_p, float u01, unsigned long long total, Target target_of, int* token) const {
    cg::cluster_group cl = cg::this_cluster();
    SfShared* lead = cl.map_shared_rank(s, 0);
    if (rank == 0) {
      int nr = 0, n = 0, lo_b[3], hi_b[3];
      unsigned long long t_lo = total, t_hi = total;                // bounds of the kept set's mass
      auto range = [&](int a, int b) {
        if (nr == 0 || lo_b[nr - 1] != a || hi_b[nr - 1] != b) {    // (the same bins again: gathered once)
          n += (int)(s->pc[b + 1] - s->pc[a]);
          lo_b[nr] = a; hi_b[nr] = b; ++nr;
        }
        t_lo = s->pm[a]; t_hi = s->pm[b + 1];
      };
      if (count_all) {
        find(s->pm, s->pc, true, (unsigned long long)(top_k - 1));
        range(s->bin, s->bin);
      }
      if (top_p < 1.0f) {
        find_two(target_of(t_lo, (double)top_p), target_of(t_hi, (double)top_p));
        range(s->at[0], s->at[1]);
        __syncthreads();                                            // (s->at is written again)
      }
      find_two(target_of(t_lo, (double)u01), target_of(t_hi, (double)u01));
      range(s->at[0], s->at[1]);
      if (n > SF_CAND) nr = 0;
      if ((int)threadIdx.x < size) {
        SfShared* o = cl.map_shared_rank(s, (int)threadIdx.x);
        o->ranges = nr;
        for (int k = 0; k < nr; ++k) { o->range_lo[k] = lo_b[k]; o->range_hi[k] = hi_b[k]; }
      }
      if (threadIdx.x == 0) s->n_cand = 0;
    }
    sf_sync(cl, size);
    const int nr = s->ranges;
    if (nr == 0) return false;
    int lo_b[3], hi_b[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) { lo_b[k] = k < nr ? s->range_lo[k] : 1; hi_b[k] = k < nr ? s->range_hi[k] : 0; }
    for_slice([&](float v, int i) {
      const float z = sf_scaled(v, inv_temp);
      const int b = bin_of(z);
      if (!((b >= lo_b[0] && b <= hi_b[0]) || (b >= lo_b[1] && b <= hi_b[1]) || (b >= lo_b[2] && b <= hi_b[2]))) return;
      if (!count_all && sf_mass(row, z) == 0) return;
      const unsigned slot = atomicAdd(&lead->n_cand, 1u);
      if (slot < SF_CAND) lead->cand[slot] = comp(sf_key(z), i);
    });
    sf_sync(cl, size);
    if (rank != 0) return true;
    const int nc = min((int)s->n_cand, SF_CAND), t = threadIdx.x;
    if (t < nc) {
      const float z = z_of(s->cand[t]);
      s->cmass[t] = sf_mass(row, z);
      s->cbin[t] = bin_of(z);
    }
    __syncthreads();
    const int c = t >> 2;
    const unsigned long long mine = c < nc ? s->cand[c] : 0ull;
    const int my_bin = c < nc ? s->cbin[c] : -1;
    unsigned long long bm = 0;
    unsigned int bc = 0;
    for (int j = t & 3; j < nc; j += 4)
      if (s->cand[j] > mine && s->cbin[j] == my_bin) { bm += s->cmass[j]; ++bc; }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) { bm += __shfl_xor_sync(0xffffffffu, bm, o); bc += __shfl_xor_sync(0xffffffffu, bc, o); }
    if (c < nc && (t & 3) == 0) { s->cbefore[c] = bm + s->pm[my_bin]; s->crank_of[c] = bc + s->pc[my_bin]; }
    if (t == 0) { s->res_comp = 0x7fffffffull; s->res_before = 0; s->res_mass = 0; }
    __syncthreads();
    auto answer = [&](bool by_count, unsigned long long target) {
      if (t < nc) {
        const unsigned long long a = s->cbefore[t], m = s->cmass[t];
        if (by_count ? (unsigned long long)s->crank_of[t] == target : a <= target && target - a < m) {
          s->res_comp = s->cand[t]; s->res_before = a; s->res_mass = m;
        }
      }
      __syncthreads();
      const unsigned long long kept = s->res_before + s->res_mass;
      __syncthreads();
      return kept;
    };
    if (count_all) total = answer(true, (unsigned long long)(top_k - 1));
    if (top_p < 1.0f) total = answer(false, target_of(total, (double)top_p));
    answer(false, target_of(total, (double)u01));
    *token = 0x7fffffff - (int)(s->res_comp & 0xffffffffu);
    return true;
  }
};

// GREEDY (temperature 0): the arg-max alone, without the histograms' shared memory and registers (two CTAs fit an SM).
template <bool GREEDY>
__global__ void __launch_bounds__(SF_THREADS, GREEDY ? 2 : 1) sample_full_kernel(const SampleFullParams p) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(16) unsigned char sf_smem[];
  SfShared& sh = *reinterpret_cast<SfShared*>(sf_smem);
  __shared__ int s_last;
  __shared__ SfBest sb;
  cg::cluster_group cl = cg::this_cluster();
  const int csize = (int)cl.num_blocks(), crank = (int)cl.block_rank();
  const int row = blockIdx.x / csize;
  if (csize > 1) sf_cluster_arrive();                       // waited for before the first store into another CTA's shared memory
  if (p.cand != nullptr) {
    // every (rank, CTA) of the decode kernel has published its candidate for this row ⇒ its logits stores landed
    const unsigned int gen_now = *reinterpret_cast<const volatile unsigned int*>(p.gen);
    const uint32_t tag = gen_now * (uint32_t)p.two_l;
    const uint2* base = p.cand + (size_t)((gen_now - 1u) & 1u) * p.tp * p.grid * p.B * 2;
    for (int c = threadIdx.x; c < p.tp * p.grid; c += SF_THREADS) {
      const uint2* q = base + ((size_t)c * p.B + row) * 2;
      unsigned spins = 0;
      for (;;) {
        uint2 a, b;
        asm volatile("ld.relaxed.sys.global.v2.u32 {%0,%1}, [%2];" : "=r"(a.x), "=r"(a.y) : "l"(q) : "memory");
        asm volatile("ld.relaxed.sys.global.v2.u32 {%0,%1}, [%2];" : "=r"(b.x), "=r"(b.y) : "l"(q + 1) : "memory");
        if (a.y == tag && b.y == tag) break;
        if (++spins > (1u << 24)) {
          printf("jllama_b200: rank %d timed out waiting for the logits of rank %d (tag %u)\n", p.rank, c / p.grid, tag);
          __trap();
        }
      }
    }
    __threadfence_system();
    __syncthreads();
  }
  SfCluster q;
  q.s = &sh; q.x = p.logits + (size_t)row * p.ld; q.V = p.V; q.inv_temp = p.inv_temp; q.rank = crank; q.size = csize;
  {
    const int per = (p.V / csize + 4) & ~3;                 // a multiple of four, csize of them cover V
    q.lo = min(p.V, crank * per);
    q.hi = min(p.V, q.lo + per);
  }
  q.vec = ((uintptr_t)q.x & 15) == 0;
  q.count_all = !GREEDY && p.top_k > 0 && p.top_k < p.V;
  // ---- best (key, ~index) of the row: the arg-max, and the maximum of the scaled logits
  if (threadIdx.x == 0) { sb.best_local = 0; sb.odd_local = 0; }
  __syncthreads();
  {
    uint32_t bk = 0;                                        // a thread's indices ascend: the first of equal keys stays
    int bi = 0x7fffffff;
    bool nan = false;
    q.for_slice<GREEDY ? 2 : 4>([&](float v, int i) {
      const float z = sf_scaled(v, p.inv_temp);
      const uint32_t key = sf_key(z);
      if (key > bk || bi == 0x7fffffff) { bk = key; bi = i; }
      if (!GREEDY) nan |= !(z == z);
    });
    unsigned long long best = bi == 0x7fffffff ? 0 : SfCluster::comp(bk, bi);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long t = __shfl_xor_sync(0xffffffffu, best, o);
      best = t > best ? t : best;
    }
    const bool any_nan = __any_sync(0xffffffffu, nan);
    if ((threadIdx.x & 31) == 0) { atomicMax(&sb.best_local, best); if (any_nan) sb.odd_local = 1; }
  }
  __syncthreads();
  if (csize > 1) sf_cluster_wait();                         // every CTA of the cluster runs: its shared memory exists
  if ((int)threadIdx.x < csize) {
    SfBest* o = cl.map_shared_rank(&sb, (int)threadIdx.x);
    o->best[crank] = sb.best_local; o->odd[crank] = sb.odd_local;
  }
  sf_sync(cl, csize);
  unsigned long long best = 0;
  bool odd = false;
  for (int r = 0; r < csize; ++r) { best = sb.best[r] > best ? sb.best[r] : best; odd |= sb.odd[r] != 0; }
  int token = 0x7fffffff - (int)(best & 0xffffffffu);
  q.zmax = SfCluster::z_of(best);
  q.row = SfRow{q.x, p.V, p.inv_temp, q.zmax, 0u, 0x7fffffff};
  if constexpr (!GREEDY) {
    // Philox of (step, row) against the total of the kept set: the same target whatever the route
    const float u01 = sf_uniform(p.seed, (unsigned)(p.step ? *p.step : 0), (unsigned)row);
    if (odd || !(fabsf(q.zmax) < INFINITY)) {
      if (crank == 0) token = sf_radix_row(q.row, p.top_k, p.top_p, u01, reinterpret_cast<unsigned long long*>(sh.cnt));
    } else {
      q.clear();
      q.for_slice([&](float v, int) {
        const float z = sf_scaled(v, p.inv_temp);
        const unsigned long long m = sf_mass(q.row, z);
        if (q.count_all || m > 0) q.add(q.bin_of(z), m);
      });
      q.merge(false);
      unsigned long long total = crank == 0 ? sh.pm[SF_BINS] : 0;
      // target of a fraction of the kept set's mass Z: max(fraction·Z, 1) − 1 (a token is kept while the mass before it is < fraction·Z)
      auto target_of = [](unsigned long long z, double fraction) -> unsigned long long {
        unsigned long long t = (unsigned long long)((double)z * fraction);
        if (t > z) t = z;
        return t > 0 ? t - 1 : 0;
      };
      if (!q.all_at_once(p.top_k, p.top_p, u01, total, target_of, &token)) {
        if (q.count_all) {
          q.select(true, (unsigned long long)(p.top_k - 1));
          if (crank == 0) total = sh.res_before + sh.res_mass;
        }
        if (p.top_p < 1.0f) {
          q.select(false, target_of(total, (double)p.top_p));
          if (crank == 0) total = sh.res_before + sh.res_mass;
        }
        q.select(false, target_of(total, (double)u01));
        if (crank == 0) token = 0x7fffffff - (int)(sh.res_comp & 0xffffffffu);
      }
    }
  }
  sf_sync(cl, csize);                                                // no CTA leaves while another may still write into its shared memory
  if (crank != 0) return;
  if (threadIdx.x == 0) {
    if (token < 0 || token >= p.V) token = 0;
    p.tok[row] = token;
  }
  if (p.next_ids == nullptr) return;
  // ---- last CTA: sequence bookkeeping of all rows
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const int prev = atomicAdd(p.ticket, 1);
    s_last = prev == p.B - 1;
    if (s_last) *p.ticket = 0;
  }
  __syncthreads();
  if (s_last) {
    __threadfence();
    __shared__ int alive;
    if (threadIdx.x == 0) alive = 0;
    __syncthreads();
    const int cl = *p.cur_len;
    for (int b = threadIdx.x; b < p.B; b += SF_THREADS) {
      int t = __ldcg(p.tok + b);
      int f = p.finished[b];
      if (f) t = p.pad;
      f = f | (t == p.eos);
      p.finished[b] = f;
      p.next_ids[b] = t;
      if (cl < p.max_len) p.sequences[(size_t)b * p.max_len + cl] = t;
      if (!f) atomicAdd(&alive, 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      *p.cur_len = cl + 1;
      *p.cache_len = *p.cache_len + 1;
      *p.step_rw = *p.step_rw + 1;
      *p.n_unfinished = alive;
    }
  }
}

}  // namespace jl

using namespace jl;

// temperature == 0 → arg-max (ties: lower index); top_k <= 0 or >= V → no top-k; top_p >= 1 → no nucleus filter.
// `cand` / `gen` (may be NULL): wait for the decode kernel of every rank first (tensor-parallel logits gathered by
// multimem.st).  `next_ids` == NULL skips the bookkeeping (selection only: tok[B]).
extern "C" JL_API int jl_sample_full(const float* logits, int B, int V, int ld, float temperature, int top_k, float top_p,
                                     unsigned long long seed, const int* step, int* tok, const void* cand,
                                     const unsigned int* gen, int tp, int rank, int num_sms, int L, int* ticket,
                                     int* next_ids, int* finished, int* sequences, int max_len, int eos, int pad,
                                     int* cur_len, int* cache_len, int* step_rw, int* n_unfinished, void* stream) {
  JL_CHECK_ARG(logits && tok && ticket && B >= 1 && V >= 1 && V <= (1 << 17) && (ld >= V || ld == 0),
               "jl_sample_full: bad arguments (V=%d must be <= 131072; ld >= V, or 0 = every row reads the same logits)", V);
  if (num_sms <= 0) num_sms = 148;
  SampleFullParams p{};
  p.logits = logits; p.V = V; p.ld = ld; p.B = B;
  const bool greedy = temperature == 0.0f;
  p.inv_temp = greedy ? 1.0f : 1.0f / temperature;
  p.top_k = top_k; p.top_p = top_p; p.seed = seed; p.step = step; p.tok = tok;
  p.cand = (const uint2*)cand; p.gen = gen; p.tp = tp; p.grid = num_sms; p.two_l = 2 * L; p.rank = rank;
  p.ticket = ticket; p.next_ids = next_ids; p.finished = finished; p.sequences = sequences;
  p.max_len = max_len; p.eos = eos; p.pad = pad;
  p.cur_len = cur_len; p.cache_len = cache_len; p.step_rw = step_rw; p.n_unfinished = n_unfinished;
  // CTAs per row: as many as leave every CTA a slice of at least 4096 logits (below that the barriers cost more than the slice) and
  // all rows' CTAs resident at once, one per SM.  Clusters of eight only where two thirds of the SMs hold them: a cluster stays within
  // one GPC, and 16 of eight did not all fit (16 rows of 128256: 51 us in clusters of eight, 38 us of four).
  // Measured, nucleus 0.95, one CTA with radix passes -> now: 1 x 8000 78 -> 18 us, 1 x 32000 177 -> 21, 4 x 128256 632 -> 27,
  // 24 x 128256 650 -> 35, 64 x 128256 645 -> 47, 200 x 128256 1062 -> 135; equal logits 27.4 ms -> 70 us.
  int C = 1;
  while (C < SF_MAX_CLUSTER && V / (2 * C) >= 4096 && (long)B * 2 * C <= (2 * C < SF_MAX_CLUSTER ? num_sms : num_sms * 2 / 3)) C *= 2;
  auto* kernel = greedy ? sample_full_kernel<true> : sample_full_kernel<false>;
  const size_t smem = greedy ? 0 : sizeof(SfShared);
  if (!greedy) JL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)B * C);
  cfg.blockDim = dim3(SF_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (C > 1) {                                               // (a grid without the attribute is one of clusters of one)
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = C;
    attr[na].val.clusterDim.y = 1;
    attr[na++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  count_launch();
  JL_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
  return JL_OK;
}

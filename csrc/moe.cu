// Mixture-of-experts routing for the hybrid decoder family: choosing experts per token, ordering the (token, choice) pairs
// by expert for the grouped linear kernels (seq_linear.cu), and the weighted sum of the experts' outputs.
//
//   route    one warp per token: scores (sigmoid or softmax of the fp32 router logits), choice scores (scores plus an optional
//            per-expert bias that only the choice sees), optional restriction to the best groups of neighbouring experts, the
//            `top` largest choice scores of what is left, weights = chosen scores over their sum (when normalised) times a
//            constant.  The last E - n_real router outputs can be identity experts (no matrices: their output is the input):
//            a chosen one is reported as expert -1 and its weight is summed per token.  Everything in fp32.
//   sort     one CTA: counts per expert, segments rounded up to whole row tiles, the sorted position of every pair, the
//            source token of every sorted row and the expert of every tile.
//   combine  y[m, :] = sum_k weight[m, k] * z[pos[m, k], :]  (+ sigmoid(gate logit[m]) * shared[m, :]).
#include <stdint.h>

#include "jllama_b200.h"
#include "seq_types.cuh"

namespace jl {

enum { SCORE_SIGMOID = 0, SCORE_SOFTMAX = 1 };

struct RouteParams {
  const float* z; int ldz;          // router logits: columns 0 .. E-1 of row m
  int M, E, top;
  int groups, keep, group_top;      // groups <= 1: every expert can be chosen; group score = sum of its group_top largest
  int score, normalise;
  float scale;
  int* idx; float* wt;              // [M][top]
  const float* bias;                // [E] fp32 added to the logits, or nullptr
  const float* choice_bias;         // [E] fp32 added to the scores for the choice (groups and top) only, or nullptr
  int n_real;                       // experts 0 .. n_real-1 have matrices; n_real .. E-1 are identity experts
  float* ident_w;                   // [M]: sum of the weights of the identity experts a token chose (n_real < E)
};

constexpr int RT_WARPS = 4;

__device__ __forceinline__ void warp_argmax(float& v, int& i) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, i, o);
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
  }
}

__global__ void __launch_bounds__(RT_WARPS * 32) moe_route_kernel(RouteParams p) {
  pdl_wait();                      // programmatic dependent launch: nothing is read before the predecessor is done
  pdl_launch_dependents();
  extern __shared__ float sm[];                                  // per warp: scores [E], work copy [E], group scores [groups]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m = blockIdx.x * RT_WARPS + warp;
  if (m >= p.M) return;
  const int ng = p.groups > 1 ? p.groups : 0;
  float* s = sm + (size_t)warp * (2 * p.E + ng);
  float* work = s + p.E;
  float* gs = work + p.E;
  const float* zr = p.z + (size_t)m * p.ldz;
  auto logit = [&](int e) { return p.bias ? zr[e] + p.bias[e] : zr[e]; };
  if (p.score == SCORE_SOFTMAX) {
    float mx = -INFINITY;
    for (int e = lane; e < p.E; e += 32) mx = fmaxf(mx, logit(e));
    mx = warp_max(mx);
    float sum = 0.0f;
    for (int e = lane; e < p.E; e += 32) { const float v = expf(logit(e) - mx); s[e] = v; sum += v; }
    sum = warp_sum(sum);
    for (int e = lane; e < p.E; e += 32) s[e] = s[e] / sum;
  } else {
    for (int e = lane; e < p.E; e += 32) s[e] = sigmoid_f(logit(e));
  }
  __syncwarp();
  for (int e = lane; e < p.E; e += 32) work[e] = p.choice_bias ? s[e] + p.choice_bias[e] : s[e];
  __syncwarp();
  if (ng) {
    const int per = p.E / ng;
    for (int g = lane; g < ng; g += 32) {                        // sum of the group's group_top largest scores
      float acc = 0.0f;
      float last = INFINITY; int last_i = -1;
      for (int t = 0; t < p.group_top && t < per; ++t) {         // t-th largest: the largest that comes after (last, last_i)
        float best = -INFINITY; int bi = -1;
        for (int j = 0; j < per; ++j) {
          const float v = work[g * per + j];
          const bool after = v < last || (v == last && j > last_i);
          if (after && (v > best || bi < 0)) { best = v; bi = j; }
        }
        if (bi < 0) break;
        acc += best; last = best; last_i = bi;
      }
      gs[g] = acc;
    }
    __syncwarp();
    for (int t = 0; t < p.keep; ++t) {                           // mark the keep best groups with -inf
      float v = -INFINITY; int gi = 0x7fffffff;
      for (int g = lane; g < ng; g += 32)
        if (gs[g] > v && gs[g] != -INFINITY) { v = gs[g]; gi = g; }
      warp_argmax(v, gi);
      __syncwarp();
      if (lane == 0 && gi != 0x7fffffff) gs[gi] = -INFINITY;
      __syncwarp();
    }
    for (int e = lane; e < p.E; e += 32)
      if (gs[e / per] != -INFINITY) work[e] = -INFINITY;           // experts outside the kept groups cannot be chosen
  }
  __syncwarp();
  float sum = 0.0f, mine = 0.0f, ident = 0.0f; int mine_i = 0;
  for (int t = 0; t < p.top; ++t) {
    float v = -INFINITY; int ei = 0x7fffffff;
    for (int e = lane; e < p.E; e += 32)
      if (work[e] > v) { v = work[e]; ei = e; }
    warp_argmax(v, ei);
    if (ei == 0x7fffffff) ei = 0;
    const float sc = s[ei];
    sum += sc;
    const int eo = ei < p.n_real ? ei : -1;                      // an identity expert has no matrices to run
    if (eo < 0) ident += sc;
    if (lane == t % 32 && t < 32) { mine = sc; mine_i = eo; }
    if (t >= 32 && lane == 0) { p.idx[(size_t)m * p.top + t] = eo; p.wt[(size_t)m * p.top + t] = sc; }    // weights scaled below
    __syncwarp();
    if (lane == 0) work[ei] = -INFINITY;
    __syncwarp();
  }
  const float mul = (p.normalise ? 1.0f / (sum + 1e-20f) : 1.0f) * p.scale;
  if (lane < p.top) { p.idx[(size_t)m * p.top + lane] = mine_i; p.wt[(size_t)m * p.top + lane] = mine * mul; }
  if (p.top > 32 && lane == 0)
    for (int t = 32; t < p.top; ++t) p.wt[(size_t)m * p.top + t] *= mul;
  if (p.ident_w && lane == 0) p.ident_w[m] = ident * mul;
}

// One CTA orders the n = M * top pairs by expert.  counts / offsets live in shared memory (E + 1 ints each).
constexpr int MS_KEEP = 16;

template <int KEEP>
__global__ void __launch_bounds__(1024) moe_sort_kernel(const int* __restrict__ idx, int n, int top, int E, int tile, int cap,
                                                        int* __restrict__ pos, int* __restrict__ row_src,
                                                        int* __restrict__ tile_group, int* __restrict__ tiles_used) {
  pdl_wait();                      // programmatic dependent launch: nothing is read before the predecessor is done
  pdl_launch_dependents();
  extern __shared__ int si[];
  int* count = si;                 // [E]
  int* start = si + E;             // [E + 1], in rows
  // One CTA, so what counts is its chain of latencies: up to KEEP pairs a thread stay in registers with their ranks (all their experts
  // asked for at once), a warp adds up the counts.  2048 tokens x 4 of 32 experts: 11.4 -> 8.7 us.  KEEP is the smallest of 1, 4 and MS_KEEP that holds the
  // pairs: sixteen steps of which fifteen have nothing to do are a us (200 tokens x 2 of 8 experts: 2.8 us with pairs in memory, 3.8 with MS_KEEP, 2.6 with 1).
  const bool keep = n <= KEEP * (int)blockDim.x;
  int ex[KEEP], rank[KEEP];
  if (keep) {
#pragma unroll
    for (int u = 0; u < KEEP; ++u) {
      const int i = threadIdx.x + u * blockDim.x;
      ex[u] = i < n ? idx[i] : -1;
    }
  }
  for (int e = threadIdx.x; e < E; e += blockDim.x) count[e] = 0;
  for (int i = threadIdx.x; i < cap; i += blockDim.x) row_src[i] = -1;
  for (int i = threadIdx.x; i < cap / tile; i += blockDim.x) tile_group[i] = -1;
  __syncthreads();
  if (keep) {                                                      // rank within its expert (expert < 0: a pair that runs no expert)
#pragma unroll
    for (int u = 0; u < KEEP; ++u) rank[u] = ex[u] >= 0 ? atomicAdd(&count[ex[u]], 1) : -1;
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) pos[i] = idx[i] >= 0 ? atomicAdd(&count[idx[i]], 1) : -1;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int per = (E + 31) / 32, e0 = min(E, (int)threadIdx.x * per), e1 = min(E, e0 + per);
    int sum = 0;
    for (int e = e0; e < e1; ++e) sum += (count[e] + tile - 1) / tile * tile;
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if ((int)threadIdx.x >= o) incl += t;
    }
    int at = incl - sum;
    for (int e = e0; e < e1; ++e) { start[e] = at; at += (count[e] + tile - 1) / tile * tile; }
    if (threadIdx.x == 31) {
      start[E] = incl;
      if (tiles_used) *tiles_used = incl / tile;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x)
    for (int t = start[e] / tile; t < start[e + 1] / tile; ++t) tile_group[t] = e;
  if (keep) {
#pragma unroll
    for (int u = 0; u < KEEP; ++u) {
      const int i = threadIdx.x + u * blockDim.x;
      if (i >= n) break;
      const int at = ex[u] >= 0 ? start[ex[u]] + rank[u] : -1;     // (-1: the combine pass skips the pair)
      pos[i] = at;
      if (at >= 0) row_src[at] = i / top;
    }
    return;
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    if (idx[i] < 0) continue;                                      // pos stays -1: the combine pass skips the pair
    const int at = start[idx[i]] + pos[i];
    pos[i] = at;
    row_src[at] = i / top;
  }
}

template <typename T>
__global__ void __launch_bounds__(256) moe_combine_kernel(const float* __restrict__ z, int ldz, const int* __restrict__ pos,
                                                          const float* __restrict__ wt, int top, const float* __restrict__ shared,
                                                          int lds, const float* __restrict__ gate, int ldg,
                                                          float* __restrict__ out, int W, const int* __restrict__ idx,
                                                          const float* __restrict__ ident_w, const T* __restrict__ x, int ldx,
                                                          int vec) {
  pdl_wait();                      // programmatic dependent launch: nothing is read before the predecessor is done
  pdl_launch_dependents();
  const size_t m = blockIdx.x;
  const float g = shared ? (gate ? sigmoid_f(gate[m * ldg]) : 1.0f) : 0.0f;
  // Bounded by the bytes of z: at most eight experts' rows are known before the columns, and a thread asks for 16 bytes of each
  // before it adds the first (same order of sums).  One float at a time behind its row's index took 29 us for 2048 tokens of
  // 2048 over 4 experts (100 MB, 3.5 TB/s), then 27 (21 with 128 threads a row): the product that wrote z leaves tens of MB in L2 to be written back meanwhile.
  if (vec) {
    size_t r[8];
    float wk[8];
    bool on[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      on[k] = k < top && !(idx && idx[m * top + k] < 0);
      r[k] = on[k] ? (pos ? (size_t)pos[m * top + k] : m * top + k) * ldz : 0;
      wk[k] = on[k] ? wt[m * top + k] : 0.0f;
    }
    const float iw = ident_w ? ident_w[m] : 0.0f;
    for (int i = threadIdx.x * 4; i < W; i += blockDim.x * 4) {
      float v[8][4], sv[4], xv[4], acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (on[k]) load4(z + r[k] + i, v[k]);
      if (ident_w) load4(x + m * ldx + i, xv);
      if (shared) load4(shared + m * lds + i, sv);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (on[k]) {
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[e] = fmaf(wk[k], v[k][e], acc[e]);
        }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (ident_w) acc[e] = fmaf(iw, xv[e], acc[e]);
        if (shared) acc[e] = fmaf(g, sv[e], acc[e]);
      }
      store4(out + m * W + i, acc);
    }
    return;
  }
  for (int i = threadIdx.x; i < W; i += blockDim.x) {
    float acc = 0.0f;
    for (int k = 0; k < top; ++k) {
      if (idx && idx[m * top + k] < 0) continue;                   // an identity expert: its share comes with ident_w below
      const size_t r = pos ? (size_t)pos[m * top + k] : m * top + k;
      acc = fmaf(wt[m * top + k], z[r * ldz + i], acc);
    }
    if (ident_w) acc = fmaf(ident_w[m], to_f(x[m * ldx + i]), acc);
    if (shared) acc = fmaf(g, shared[m * lds + i], acc);
    out[m * W + i] = acc;
  }
}

// xs[p, :] = x[row_src[p], :] (row_src[p] < 0: zeros): the rows of a step in sorted order, for kernels that cannot gather.
// A CTA takes GR_ROWS of them, a thread a 16-byte column of each: the rows' loads are in flight together (a CTA per row: 14.2 us for 12256 rows of 2048
// bfloat16, 50 MB written; now 9.2).  Few rows that fill a CTA each go one to a CTA, which then are enough to fill the SMs (2176 rows of 2048: 2.9 us, four to a
// CTA 3.7; 4992 rows: 5.9 and 4.7; 2176 rows of 512: 2.8 and 1.6).
constexpr int GR_ROWS = 4;

template <typename T, int ROWS>
__global__ void __launch_bounds__(256) moe_gather_kernel(const T* __restrict__ x, int ldx, const int* __restrict__ row_src,
                                                         T* __restrict__ xs, int rows, int W) {
  pdl_wait();                      // programmatic dependent launch: nothing is read before the predecessor is done
  pdl_launch_dependents();
  const size_t p = (size_t)blockIdx.x * ROWS;
  int src[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) src[r] = p + r < (size_t)rows ? row_src[p + r] : -1;
  constexpr int VN = 16 / sizeof(T);
  if (W % VN == 0 && ldx % VN == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)xs & 15) == 0) {
    for (int i = threadIdx.x; i < W / VN; i += blockDim.x) {
      uint4 v[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
        v[r] = src[r] >= 0 ? reinterpret_cast<const uint4*>(x + (size_t)src[r] * ldx)[i] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
        if (p + r < (size_t)rows) reinterpret_cast<uint4*>(xs + (p + r) * W)[i] = v[r];
    }
    return;
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    if (p + r >= (size_t)rows) break;
    for (int i = threadIdx.x; i < W; i += blockDim.x) xs[(p + r) * W + i] = src[r] >= 0 ? x[(size_t)src[r] * ldx + i] : from_f<T>(0.0f);
  }
}

}  // namespace jl

using namespace jl;

// 16-byte columns for moe_combine_kernel: every row it reads starts on a 16-byte boundary (x: 8 bytes, four 16-bit numbers)
static int combine_vec(const float* z, int ldz, int top, const float* shared, int lds, const float* out, int W, const void* x, int ldx) {
  return top <= 8 && W % 4 == 0 && ldz % 4 == 0 && (shared == nullptr || lds % 4 == 0) && (x == nullptr || ldx % 4 == 0) &&
         ((uintptr_t)z | (uintptr_t)shared | (uintptr_t)out | (uintptr_t)x) % 16 == 0;
}

// Threads of a row: 128 where the rows fill every SM four times over, because a thread's rows then wait behind one look at the indices (2048
// tokens x 4 experts, 2048 columns: 256 threads 26 us, 128 21, 512 35; 600 x 2 x 4096: 20.5 and 16.4); with fewer rows the columns' parallelism
// counts (200 x 4 x 2048: 256 threads 10.2, 128 11.2; 64 x 4 x 4096 10.2 and 14.3).
static int combine_threads(int M, int vec) { return vec && M >= 4 * SMS ? 128 : 256; }

static int moe_route_launch(const float* z, int ldz, int M, int E, int top, int groups, int keep, int group_top, int score,
                            int normalise, float scale, const float* bias, const float* choice_bias, int n_real, float* ident_w,
                            int* idx, float* wt, void* stream) {
  JL_CHECK_ARG(M >= 1 && E >= 1 && top >= 1 && top <= E && ldz >= E, "jl_moe_route: bad shape M=%d E=%d top=%d ldz=%d", M, E, top, ldz);
  JL_CHECK_ARG(groups <= 1 || (E % groups == 0 && keep >= 1 && keep <= groups && group_top >= 1 && keep * (E / groups) >= top),
               "jl_moe_route: %d groups of %d experts, keep %d, cannot give %d choices", groups, groups > 0 ? E / groups : 0, keep, top);
  JL_CHECK_ARG(score == SCORE_SIGMOID || score == SCORE_SOFTMAX, "jl_moe_route: score function %d", score);
  JL_CHECK_ARG(n_real >= 1 && n_real <= E && (n_real == E || ident_w != nullptr), "jl_moe_route: %d of %d experts with matrices", n_real, E);
  RouteParams p{z, ldz, M, E, top, groups, keep, group_top, score, normalise, scale, idx, wt, bias, choice_bias, n_real, ident_w};
  const size_t smem = (size_t)RT_WARPS * (2 * E + (groups > 1 ? groups : 0)) * sizeof(float);
  JL_CHECK_ARG(smem <= 200 * 1024, "jl_moe_route: %d experts do not fit shared memory", E);
  if (smem > 48 * 1024) JL_CUDA(cudaFuncSetAttribute(moe_route_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  JL_LAUNCH_PDL(moe_route_kernel, dim3((M + RT_WARPS - 1) / RT_WARPS), dim3(RT_WARPS * 32), smem, stream, p);
  JL_CUDA(cudaGetLastError());
  return JL_OK;
}

extern "C" JL_API int jl_moe_route(const float* z, int ldz, int M, int E, int top, int groups, int keep, int group_top, int score,
                                   int normalise, float scale, const float* bias, int* idx, float* wt, void* stream) {
  return moe_route_launch(z, ldz, M, E, top, groups, keep, group_top, score, normalise, scale, bias, nullptr, E, nullptr, idx, wt, stream);
}

// The same with a choice bias (added to the scores for groups and top only) and identity experts: router outputs n_real .. E-1
// have no matrices; a chosen one is reported as expert -1 and its weight is added to ident_w[m].
extern "C" JL_API int jl_moe_route_ex(const float* z, int ldz, int M, int E, int top, int groups, int keep, int group_top, int score,
                                      int normalise, float scale, const float* bias, const float* choice_bias, int n_real,
                                      float* ident_w, int* idx, float* wt, void* stream) {
  return moe_route_launch(z, ldz, M, E, top, groups, keep, group_top, score, normalise, scale, bias, choice_bias, n_real, ident_w, idx,
                          wt, stream);
}

// Rows of the sorted layout for n pairs over E experts with row tiles of `tile`: every expert's segment is rounded up.
extern "C" JL_API int jl_moe_sorted_rows(int n, int E, int tile) { return (n + E * (tile - 1) + tile - 1) / tile * tile; }

extern "C" JL_API int jl_moe_sort(const int* idx, int M, int top, int E, int tile, int cap, int* pos, int* row_src, int* tile_group,
                                  int* tiles_used, void* stream) {
  JL_CHECK_ARG(M >= 1 && top >= 1 && E >= 1 && tile >= 1, "jl_moe_sort: bad shape");
  JL_CHECK_ARG(cap % tile == 0 && cap >= jl_moe_sorted_rows(M * top, E, tile), "jl_moe_sort: %d rows are too few", cap);
  const size_t smem = (size_t)(2 * E + 1) * sizeof(int);
  JL_CHECK_ARG(smem <= 48 * 1024, "jl_moe_sort: %d experts do not fit shared memory", E);
  const int n = M * top;
  auto* kernel = n <= 1024 ? moe_sort_kernel<1> : n <= 4096 ? moe_sort_kernel<4> : moe_sort_kernel<MS_KEEP>;
  JL_LAUNCH_PDL(kernel, dim3(1), dim3(1024), smem, stream, idx, n, top, E, tile, cap, pos, row_src, tile_group, tiles_used);
  JL_CUDA(cudaGetLastError());
  return JL_OK;
}

extern "C" JL_API int jl_moe_combine(const float* z, int ldz, const int* pos, const float* wt, int top, const float* shared, int lds,
                                     const float* gate, int ldg, float* out, int M, int W, void* stream) {
  JL_CHECK_ARG(M >= 1 && W >= 1 && top >= 1 && ldz >= W, "jl_moe_combine: bad shape");
  const int vec = combine_vec(z, ldz, top, shared, lds, out, W, nullptr, 0);
  JL_LAUNCH_PDL(moe_combine_kernel<float>, dim3(M), dim3(combine_threads(M, vec)), 0, stream, z, ldz, pos, wt, top, shared, lds, gate, ldg, out, W,
                (const int*)nullptr, (const float*)nullptr, (const float*)nullptr, 0, vec);
  JL_CUDA(cudaGetLastError());
  return JL_OK;
}

// The same for a router with identity experts: pairs with idx < 0 ran no expert (their rows of z are not read); ident_w[m] · x[m, :]
// (x in `dtype`, row pitch ldx) is added instead.
extern "C" JL_API int jl_moe_combine_ex(const float* z, int ldz, const int* pos, const float* wt, int top, const float* shared, int lds,
                                        const float* gate, int ldg, float* out, int M, int W, const int* idx, const float* ident_w,
                                        const void* x, int ldx, int dtype, void* stream) {
  JL_CHECK_ARG(M >= 1 && W >= 1 && top >= 1 && ldz >= W, "jl_moe_combine: bad shape");
  JL_CHECK_ARG(ident_w == nullptr || (x != nullptr && ldx >= W), "jl_moe_combine: identity weights without the input rows");
  const int vec = combine_vec(z, ldz, top, shared, lds, out, W, x, ldx);
  JL_DISPATCH_DTYPE(dtype, JL_LAUNCH_PDL(moe_combine_kernel<T>, dim3(M), dim3(combine_threads(M, vec)), 0, stream, z, ldz, pos, wt, top, shared, lds, gate,
                                         ldg, out, W, idx, ident_w, (const T*)x, ldx, vec));
  JL_CUDA(cudaGetLastError());
  return JL_OK;
}

extern "C" JL_API int jl_moe_gather(const void* x, int ldx, const int* row_src, void* xs, int rows, int W, int dtype, void* stream) {
  JL_CHECK_ARG(rows >= 1 && W >= 1 && ldx >= W, "jl_moe_gather: bad shape");
  const bool few = rows <= 3072 && (long)W * (dtype == DT_BF16 ? 2 : 4) >= 2048;
  if (few)
    JL_DISPATCH_DTYPE(dtype, JL_LAUNCH_PDL((moe_gather_kernel<T, 1>), dim3(rows), dim3(128), 0, stream, (const T*)x, ldx, row_src, (T*)xs, rows, W));
  else
    JL_DISPATCH_DTYPE(dtype, JL_LAUNCH_PDL((moe_gather_kernel<T, GR_ROWS>), dim3((rows + GR_ROWS - 1) / GR_ROWS), dim3(256), 0, stream, (const T*)x, ldx,
                                           row_src, (T*)xs, rows, W));
  JL_CUDA(cudaGetLastError());
  return JL_OK;
}

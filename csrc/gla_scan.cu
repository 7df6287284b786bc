// Gated linear attention: the per-head matrix state S [D x Dv] with one decay per key channel (prompts with projected decays and up to 128 key channels: gla_chunk.cu),
//     S_t = diag(alpha_t) S_(t-1) + k_t v_t^T,     o_t = S_t^T q_t,
// advanced token by token in fp32, for prompts (S tokens per row) and for decoding (S = 1) alike.
//
// The decay comes from a low-rank projection: z = A2 (A1 h) + bias, alpha = sigmoid(z)^(1/tau) = exp(logsigmoid(z) / tau).
// The rank-R product A1 h arrives as R fp32 columns of the fused projection buffer; the A2 product, the bias, the
// log-sigmoid and the exponential are done here in fp32 for a chunk of tokens at a time.
//
// Work split: grid (value-column slices, heads, batch rows); a thread owns GS_DP = 32 key channels of one value column of
// the state in registers, P = ceil(D / 32) (rounded to a power of two) adjacent lanes share a column and add their
// partial o with shuffles.  q, k and alpha of a chunk of tokens are staged in shared memory, one row of 36 floats per
// 32 channels (16-byte loads; the P lanes of a column read different banks).  Padding tokens (slot < pad_left[b]) are skipped:
// the state of a left-padded row starts at its first real token.
#include <stdlib.h>

#include "gla_scan.cuh"
#include "jllama_b200.h"
#include "seq_types.cuh"
#include "tcgen05.cuh"

namespace jl {

constexpr int GS_DP = 32;        // state rows per thread
constexpr int GS_TC = 8;         // tokens staged per chunk
constexpr int GS_THREADS = 128;
constexpr int GS_PITCH = GS_DP + 4;   // floats per 32 channels in shared memory: 16-byte aligned rows, distinct banks per lane group


template <typename T>
__global__ void __launch_bounds__(GS_THREADS, 3) gla_scan_kernel(GlaParams p, const T* __restrict__ a2, const T* __restrict__ a2b) {
  pdl_wait();                      // programmatic dependent launch: nothing is read before the predecessor is done
  pdl_launch_dependents();
  extern __shared__ float4 smem4[];
  float* smem = reinterpret_cast<float*>(smem4);
  const int P = p.P;                                         // lanes per value column (power of two, adjacent lanes of a warp)
  const int cols = GS_THREADS / P;                           // value columns per CTA
  const int tid = threadIdx.x;
  const int part = tid % P, lcol = tid / P, col = blockIdx.x * cols + lcol;
  const int h = blockIdx.y, b = blockIdx.z;
  const int DS = P * GS_PITCH;                               // padded channel pitch of one token's q / k / alpha
  float* qs = smem;                                          // [TC][DS]
  float* ks = qs + GS_TC * DS;
  float* as = ks + GS_TC * DS;
  float* vs = as + GS_TC * DS;                               // [TC][cols]
  float* zs = vs + GS_TC * cols;                             // [TC][R]

  const bool idle = (int)blockIdx.x * cols + (tid & ~31) / P >= p.Dv;      // warp-uniform: no column of this warp exists
  float st[GS_DP];
  const int d0 = part * GS_DP;
  float* sbase = p.state + (((size_t)b * p.H + h) * p.D) * p.Dv;
#pragma unroll
  for (int r = 0; r < GS_DP; ++r) st[r] = (col < p.Dv && d0 + r < p.D) ? sbase[(size_t)(d0 + r) * p.Dv + col] : 0.0f;

  const int first = max(0, (p.pad_left ? p.pad_left[b] : 0) - (p.cache_len ? *p.cache_len : 0));   // first real token of this call
  if (part == 0 && col < p.Dv)                               // padding tokens: defined (zero) output rows
    for (int s = 0; s < min(first, p.S); ++s) p.o[((size_t)(b * p.S + s) * p.H + h) * p.Dv + col] = 0.0f;
  for (int s0 = first; s0 < p.S; s0 += GS_TC) {
    const int nt = min(GS_TC, p.S - s0);
    __syncthreads();
    for (int i = tid; i < nt * p.R; i += GS_THREADS) {
      const int t = i / p.R, r = i % p.R;
      zs[t * p.R + r] = p.y[(size_t)(b * p.S + s0 + t) * p.ldy + p.a_off + r];
    }
    for (int i = tid; i < nt * cols; i += GS_THREADS) {
      const int t = i / cols, c = blockIdx.x * cols + i % cols;
      vs[i] = scan_value(p, (size_t)(b * p.S + s0 + t), h, c);
    }
    __syncthreads();
    for (int i = tid; i < nt * P * GS_DP; i += GS_THREADS) {
      const int t = i / (P * GS_DP), d = i % (P * GS_DP);
      const int at = t * DS + (d / GS_DP) * GS_PITCH + d % GS_DP;
      float qv = 0.0f, kv = 0.0f, av = 1.0f;
      if (d < p.D)
        scan_channel<T>(p, (size_t)(b * p.S + s0 + t), h, d, scan_position(p, b, s0 + t), zs + t * p.R, a2, a2b, qv, kv, av);
      qs[at] = qv; ks[at] = kv; as[at] = av;
    }
    __syncthreads();
    if (idle) continue;
    for (int t = 0; t < nt; ++t) {
      const float v = vs[t * cols + lcol];
      const float4* qt = reinterpret_cast<const float4*>(qs + t * DS + part * GS_PITCH);
      const float4* kt = reinterpret_cast<const float4*>(ks + t * DS + part * GS_PITCH);
      const float4* at = reinterpret_cast<const float4*>(as + t * DS + part * GS_PITCH);
      float a0 = 0.0f, a1 = 0.0f, a2v = 0.0f, a3 = 0.0f;
#pragma unroll
      for (int r = 0; r < GS_DP / 4; ++r) {
        const float4 al = at[r], kk = kt[r], qq = qt[r];
        st[4 * r + 0] = fmaf(al.x, st[4 * r + 0], kk.x * v); a0 = fmaf(qq.x, st[4 * r + 0], a0);
        st[4 * r + 1] = fmaf(al.y, st[4 * r + 1], kk.y * v); a1 = fmaf(qq.y, st[4 * r + 1], a1);
        st[4 * r + 2] = fmaf(al.z, st[4 * r + 2], kk.z * v); a2v = fmaf(qq.z, st[4 * r + 2], a2v);
        st[4 * r + 3] = fmaf(al.w, st[4 * r + 3], kk.w * v); a3 = fmaf(qq.w, st[4 * r + 3], a3);
      }
      float acc = (a0 + a1) + (a2v + a3);
      for (int off = P >> 1; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
      if (part == 0 && col < p.Dv) p.o[((size_t)(b * p.S + s0 + t) * p.H + h) * p.Dv + col] = acc;
    }
  }
#pragma unroll
  for (int r = 0; r < GS_DP; ++r)
    if (col < p.Dv && d0 + r < p.D) sbase[(size_t)(d0 + r) * p.Dv + col] = st[r];
}


// One token per row, with the head norm and the gate behind it (jl_gla_step): a CTA has a whole head, a thread DP key channels of one value column, so
// that the read-outs meet in shared memory and leave normed, gated and in the operand type.  What bounds such a step is latency: the state (asked for into
// L2 while the projection before still runs), the projection's row, the decays and the two sums.  One launch for the scan's and the norm's, us in a graph: 16 heads of 64 x
// 128, 1 and 2 rows 6.6 -> 4.2, 8 rows 7.4 -> 4.2, 64 rows 28.1 -> 16.8; 8 heads of 128 x 128, 2 rows 7.0 -> 6.1, 64 rows 31.3 -> 15.5.
struct GlaStep {
  GlaParams p;
  int g_off;                           // gate columns of y
  float eps;
  int gate_act;
};

template <typename T, int DP>
__global__ void __launch_bounds__(1024) gla_step_kernel(const GlaStep a, const T* __restrict__ a2, const T* __restrict__ a2b, const T* __restrict__ norm,
                                                        T* __restrict__ out) {
  const GlaParams& p = a.p;
  extern __shared__ float4 smem4[];
  __shared__ float red[33];
  const int cols = (p.Dv + 31) & ~31, P = blockDim.x / cols, D4 = P * DP;      // value columns in whole warps; channels in whole parts
  float* qs = reinterpret_cast<float*>(smem4);                 // q | k | alpha [D4], then the partial read-outs [P][cols]
  float* ks = qs + D4;
  float* as = ks + D4;
  float* part_o = as + D4;
  const int tid = threadIdx.x, part = tid / cols, col = tid % cols, h = blockIdx.x, b = blockIdx.y;
  float* sbase = p.state + ((size_t)b * p.H + h) * p.D * p.Dv;
  for (int i = tid * 32; i < p.D * p.Dv; i += blockDim.x * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(sbase + i));
  pdl_wait();                      // nothing is read before the predecessor is done (the prefetch above returns nothing)
  pdl_launch_dependents();
  const bool real = (p.pad_left ? p.pad_left[b] : 0) <= (p.cache_len ? *p.cache_len : 0);
  const float* yr = p.y + (size_t)b * p.ldy;
  const bool on = col < p.Dv;
  const int cc = min(col, p.Dv - 1), d0 = part * DP;
  float st[DP];
#pragma unroll
  for (int r = 0; r < DP; ++r) st[r] = d0 + r < p.D ? sbase[(size_t)(d0 + r) * p.Dv + cc] : 0.0f;
  const float v = yr[p.v_off + h * p.Dv + cc], gate = yr[a.g_off + h * p.Dv + cc], w = norm ? to_f(norm[cc]) : 1.0f;
  for (int d = tid; d < D4; d += blockDim.x) {
    float qv = 0.0f, kv = 0.0f, av = 1.0f;
    if (d < p.D) {
      const int n = h * p.D + d;
      qv = yr[p.q_off + n] * p.q_scale;
      kv = yr[p.k_off + n] * p.k_scale;
      float z = to_f(a2b[n]);
      for (int r = 0; r < p.R; r += 8) {                       // (all loads of a round first, the sum in order of r)
        float wv[8], zv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int rr = min(r + u, p.R - 1);
          wv[u] = to_f(a2[(size_t)n * p.R + rr]);
          zv[u] = yr[p.a_off + rr];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) if (r + u < p.R) z = fmaf(wv[u], zv[u], z);
      }
      av = expf(log_sigmoid(z) * p.inv_tau);
    }
    qs[d] = qv; ks[d] = kv; as[d] = av;
  }
  __syncthreads();
  float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int r = 0; r < DP; ++r) {
    st[r] = fmaf(as[d0 + r], st[r], ks[d0 + r] * v);
    acc[r & 3] = fmaf(qs[d0 + r], st[r], acc[r & 3]);
  }
  part_o[part * cols + col] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
  if (real && on) {
#pragma unroll
    for (int r = 0; r < DP; ++r)
      if (d0 + r < p.D) sbase[(size_t)(d0 + r) * p.Dv + col] = st[r];
  }
  __syncthreads();
  float o = 0.0f;
  if (part == 0 && on && real)                                 // (a padding token: a zero row, the state as it was)
    for (int q = 0; q < P; ++q) o += part_o[q * cols + col];
  const float r = 1.0f / sqrtf(block_sum(o * o, red) / (float)p.Dv + a.eps);
  if (part == 0 && on) out[((size_t)b * p.H + h) * p.Dv + col] = from_f<T>(o * r * w * apply_act(gate, a.gate_act, 0.0f, 0.0f));
}

// ---------------------------------------------------------------------------------------------------------------------
// Prompts: the same recurrence in two launches.  gla_prep_kernel is token-parallel: it forms alpha (low-rank product,
// bias, log-sigmoid, exponential — fp32), scales q, and writes q | k | alpha | v of every (token, head) as one
// contiguous fp32 record laid out exactly like the scan's shared-memory stage ([3][P][DP + 4] then the value row,
// padded to 16 bytes).  In gla_stream_kernel one thread copies records with bulk copies, two stages deep (the copy of the next
// GS_TS tokens runs under the arithmetic of the current ones), and all advance the state.  The fused kernel above pays two
// dependent DRAM round trips and the transcendental math per 8 tokens on the critical path of a sequential loop; here
// the loop sees shared memory only.
//
// A thread of the streaming kernel owns a DP x C = 16 x 4 tile of the state: 16 key channels of 4 adjacent value columns, the P = D / 16
// lanes of a column group adjacent.  What bounds the loop is the path from shared memory to registers (128 bytes a cycle and SM,
// broadcast or not): q, k and alpha of a thread's channels are read once for its four columns, 12 reads of 16 bytes per token for 64
// state elements (the former 32 x 1 tile: 24 reads for 32), and channels go in pairs through packed fp32 instructions
// (fma.rn.f32x2: two rounded FMAs), three for two state elements of one token.  A group's partial read-outs meet by
// exchanging halves: P = 4 lanes need three shuffles for four columns and end with one column each.
// 2048 tokens, 16 heads of 64 x 128, one row on one B200, both passes: 189 us with the 32 x 1 tile, 93 us with this one.
constexpr int GS_TS = 16;        // tokens per pipeline stage
constexpr int GT_DP = 16, GT_C = 4, GT_PITCH = GT_DP + 4;      // 16 channels in rows of 20 floats: the lanes of a group read different banks
constexpr int GT_MAX_D = 256;    // wider keys: the fused kernel above

__host__ __device__ inline int gla_lanes(int D) {
  int P = 1;
  while (P * GT_DP < D) P *= 2;
  return P;
}
// threads of a CTA: whole warps that cover the value columns, at most 128
inline int gla_threads(int P, int Dv) {
  const int t = ((Dv + GT_C - 1) / GT_C * P + 31) / 32 * 32;
  return t < GS_THREADS ? t : GS_THREADS;
}
__host__ __device__ inline int gla_record_floats(int P, int Dv) { return 3 * P * GT_PITCH + ((Dv + 3) & ~3); }

// Whether the preparation's options are all off: q, k and v as they lie in y, the decay projected, its rows of A2 in whole pieces of 16 bytes (at
// most GP_PIECES).  The instance for these calls (PLAIN) is a small part of the general one's code and asks for all that a thread needs at once, before the
// barrier: 2048 tokens of 16 heads (64 / 128, rank 16) 42 -> 25 us, where 100 MB read and written take 15.
constexpr int GP_PIECES = 4;
inline bool gla_plain(const GlaParams& p, const void* a2, int elem) {
  return p.rot == 0 && p.act == ACT_NONE && p.aux == nullptr && p.head_decay == nullptr && p.ones == 0 && p.qk_div <= 1 &&
         p.R * elem % 16 == 0 && p.R * elem <= 16 * GP_PIECES && ((uintptr_t)a2 & 15) == 0;
}

// A thread forms one slot of the records (a channel of a head, or a value column) for GP_TOK tokens: the channel's row of A2 is read once
// for all of them.  (One CTA per token, its threads walking all channels, read A2 once per token: 60 us for 2048 tokens of 16 x 64 channels
// against 42 us in the general instance.)
constexpr int GP_TOK = 8, GP_THREADS = 256;

template <typename T, bool PLAIN>
__global__ void __launch_bounds__(GP_THREADS) gla_prep_kernel(GlaParams p, const T* __restrict__ a2, const T* __restrict__ a2b,
                                                              float* __restrict__ rec) {
  pdl_wait();                      // programmatic dependent launch: nothing is read before the predecessor is done
  pdl_launch_dependents();
  extern __shared__ float4 zs4[];                               // [GP_TOK][R]
  float* zs = reinterpret_cast<float*>(zs4);
  const int M = p.B * p.S, m0 = blockIdx.x * GP_TOK, nt = min(GP_TOK, M - m0);
  if constexpr (PLAIN) {
    const int P = p.P, RF = gla_record_floats(P, p.Dv), per_head = P * GT_DP, dvp = (p.Dv + 3) & ~3;
    const int i = blockIdx.y * GP_THREADS + threadIdx.x, nq = p.H * per_head;
    const bool value = i >= nq;
    const int j = value ? i - nq : i, h = value ? j / dvp : j / per_head, d = value ? j % dvp : j % per_head;
    const bool on = value ? h < p.H && d < p.Dv : d < p.D;
    const float* src = p.y + (size_t)m0 * p.ldy + (value ? p.v_off + h * p.Dv : p.q_off + h * p.D) + d;
    const float* ksrc = p.y + (size_t)m0 * p.ldy + p.k_off + h * p.D + d;
    float qv[GP_TOK], kv[GP_TOK], av[GP_TOK];
    constexpr int N = 16 / sizeof(T);
    uint4 row[GP_PIECES];
    float bias = 0.0f;
#pragma unroll
    for (int t = 0; t < GP_TOK; ++t) qv[t] = on && t < nt ? src[(size_t)t * p.ldy] : 0.0f;
    if (on && !value) {
#pragma unroll
      for (int t = 0; t < GP_TOK; ++t) kv[t] = t < nt ? ksrc[(size_t)t * p.ldy] : 0.0f;
      const int n = h * p.D + d;
      bias = to_f(a2b[n]);
#pragma unroll
      for (int u = 0; u < GP_PIECES; ++u)
        if (u * N < p.R) row[u] = *reinterpret_cast<const uint4*>(a2 + (size_t)n * p.R + u * N);
    }
    for (int e = threadIdx.x; e < GP_TOK * p.R; e += GP_THREADS)
      zs[e] = e < nt * p.R ? p.y[(size_t)(m0 + e / p.R) * p.ldy + p.a_off + e % p.R] : 0.0f;
    __syncthreads();
    if (value) {
      if (h >= p.H) return;
      float* out = rec + ((size_t)m0 * p.H + h) * RF + 3 * P * GT_PITCH + d;
#pragma unroll
      for (int t = 0; t < GP_TOK; ++t) if (t < nt) out[(size_t)t * p.H * RF] = qv[t];
      return;
    }
#pragma unroll
    for (int t = 0; t < GP_TOK; ++t) av[t] = bias;
    if (on) {
#pragma unroll
      for (int u = 0; u < GP_PIECES; ++u) {
        if (u * N >= p.R) break;
        const T* e = reinterpret_cast<const T*>(&row[u]);
#pragma unroll
        for (int c = 0; c < N; c += 4)
#pragma unroll
          for (int t = 0; t < GP_TOK; ++t) {
            const float4 z = zs4[(t * p.R + u * N + c) >> 2];
            av[t] = fmaf(to_f(e[c]), z.x, av[t]);
            av[t] = fmaf(to_f(e[c + 1]), z.y, av[t]);
            av[t] = fmaf(to_f(e[c + 2]), z.z, av[t]);
            av[t] = fmaf(to_f(e[c + 3]), z.w, av[t]);
          }
      }
#pragma unroll
      for (int t = 0; t < GP_TOK; ++t) av[t] = expf(log_sigmoid(av[t]) * p.inv_tau);
    }
    float* out = rec + ((size_t)m0 * p.H + h) * RF + (d / GT_DP) * GT_PITCH + d % GT_DP;
#pragma unroll
    for (int t = 0; t < GP_TOK; ++t) {
      if (t >= nt) break;
      float* o = out + (size_t)t * p.H * RF;
      o[0] = on ? qv[t] * p.q_scale : 0.0f; o[P * GT_PITCH] = on ? kv[t] * p.k_scale : 0.0f; o[2 * P * GT_PITCH] = on ? av[t] : 1.0f;
    }
    return;
  }
  for (int i = threadIdx.x; i < nt * p.R; i += GP_THREADS) zs[i] = p.y[(size_t)(m0 + i / p.R) * p.ldy + p.a_off + i % p.R];
  __syncthreads();
  const int P = p.P, RF = gla_record_floats(P, p.Dv), per_head = P * GT_DP, dvp = (p.Dv + 3) & ~3;
  const int i = blockIdx.y * GP_THREADS + threadIdx.x;
  if (i >= p.H * per_head) {                                    // a value column
    const int j = i - p.H * per_head;
    if (j >= p.H * dvp) return;
    const int h = j / dvp, c = j % dvp;
    float* out = rec + ((size_t)m0 * p.H + h) * RF + 3 * P * GT_PITCH + c;
    float v[GP_TOK];
#pragma unroll
    for (int t = 0; t < GP_TOK; ++t) v[t] = t < nt ? scan_value(p, (size_t)(m0 + t), h, c) : 0.0f;
#pragma unroll
    for (int t = 0; t < GP_TOK; ++t) if (t < nt) out[(size_t)t * p.H * RF] = v[t];
    return;
  }
  const int h = i / per_head, d = i % per_head;
  float* out = rec + ((size_t)m0 * p.H + h) * RF + (d / GT_DP) * GT_PITCH + d % GT_DP;
  float qv[GP_TOK], kv[GP_TOK], av[GP_TOK];
#pragma unroll
  for (int t = 0; t < GP_TOK; ++t) { qv[t] = kv[t] = 0.0f; av[t] = 1.0f; }
  if (d < p.D) {
#pragma unroll
    for (int t = 0; t < GP_TOK; ++t)
      if (t < nt) scan_qk(p, (size_t)(m0 + t), h, d, scan_position(p, (m0 + t) / p.S, (m0 + t) % p.S), qv[t], kv[t]);
    if (p.aux || p.head_decay) {
#pragma unroll
      for (int t = 0; t < GP_TOK; ++t) if (t < nt) av[t] = p.aux ? p.aux[(size_t)(m0 + t) * p.ld_aux + h] : p.head_decay[h];
    } else {
      const int n = h * p.D + d;
      const float bias = to_f(a2b[n]);
#pragma unroll
      for (int t = 0; t < GP_TOK; ++t) av[t] = bias;
      for (int r = 0; r < p.R; ++r) {
        const float a = to_f(a2[(size_t)n * p.R + r]);
#pragma unroll
        for (int t = 0; t < GP_TOK; ++t) av[t] = fmaf(a, t < nt ? zs[t * p.R + r] : 0.0f, av[t]);
      }
#pragma unroll
      for (int t = 0; t < GP_TOK; ++t) av[t] = expf(log_sigmoid(av[t]) * p.inv_tau);
    }
  }
#pragma unroll
  for (int t = 0; t < GP_TOK; ++t) {
    if (t >= nt) break;
    float* o = out + (size_t)t * p.H * RF;
    o[0] = qv[t]; o[P * GT_PITCH] = kv[t]; o[2 * P * GT_PITCH] = av[t];
  }
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, int bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void fence_generic_to_bulk() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ unsigned long long f2_dup(float v) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float2 f2_split(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ unsigned long long f2_join(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}

// P lanes of a column group; MODE 0: one chunk, state in / out; 1: local scan of a chunk from zero, no read-out; 3: read-out pass
template <int P, int MODE>
__global__ void __launch_bounds__(GS_THREADS, 3) gla_stream_kernel(GlaParams p, const float* __restrict__ rec) {
  pdl_wait();                      // programmatic dependent launch: nothing is read before the predecessor is done
  pdl_launch_dependents();
  extern __shared__ float4 smem4[];
  __shared__ __align__(8) unsigned long long bars[2];
  float* smem = reinterpret_cast<float*>(smem4);
  const int nthreads = blockDim.x, cols = nthreads / P * GT_C;          // value columns per CTA
  const int tid = threadIdx.x, part = tid % P, grp = tid / P;
  const int col0 = blockIdx.x * cols + grp * GT_C;                      // first of this thread's columns
  const int h = blockIdx.y, b = blockIdx.z / p.NC, chunk = blockIdx.z % p.NC;
  const bool idle = (int)blockIdx.x * cols + (tid & ~31) / P * GT_C >= p.Dv;      // warp-uniform: no column of this warp exists
  constexpr int QKA = 3 * P * GT_PITCH;                                 // floats of q | k | alpha per token
  const int SF = QKA + cols;                                            // floats per token in a stage
  const int RF = gla_record_floats(P, p.Dv);
  const bool vec = p.Dv % 4 == 0 && ((uintptr_t)(MODE == 0 ? p.state : p.cstate) & 15) == 0;      // rows of the state on 16-byte boundaries
  unsigned long long st[GT_DP / 2][GT_C];                               // pairs of channels
  const int d0 = part * GT_DP;
  float* sbase = MODE == 0 ? p.state + (((size_t)b * p.H + h) * p.D) * p.Dv
                           : p.cstate + ((((size_t)b * p.NC + chunk) * p.H + h) * p.D) * p.Dv;
  auto load_row = [&](int r, float (&v)[GT_C]) {
    const float* src = sbase + (size_t)(d0 + r) * p.Dv + col0;
    if (MODE == 1 || d0 + r >= p.D || col0 >= p.Dv) {
#pragma unroll
      for (int c = 0; c < GT_C; ++c) v[c] = 0.0f;
    } else if (vec) {
      load4(src, v);
    } else {
#pragma unroll
      for (int c = 0; c < GT_C; ++c) v[c] = col0 + c < p.Dv ? src[c] : 0.0f;
    }
  };
#pragma unroll
  for (int r = 0; r < GT_DP; r += 2) {
    float v0[GT_C], v1[GT_C];
    load_row(r, v0);
    load_row(r + 1, v1);
#pragma unroll
    for (int c = 0; c < GT_C; ++c) st[r / 2][c] = f2_join(v0[c], v1[c]);
  }
  const bool decays = MODE == 1 && blockIdx.x == 0 && (tid & ~31) == 0;  // warp-uniform: this warp multiplies up the chunk's decays
  unsigned long long ap[GT_DP / 2];
#pragma unroll
  for (int r = 0; r < GT_DP / 2; ++r) ap[r] = f2_dup(1.0f);
  // columns of a finished read-out that this lane holds after the exchange, and whether it writes them
  constexpr int NOUT = P == 1 ? 4 : (P == 2 ? 2 : 1), REST = P >= 4 ? P / 4 - 1 : 0;
  const int ocol = col0 + (P >= 2 && (part & (P / 2)) ? 2 : 0) + (P >= 4 && (part & (P / 4)) ? 1 : 0);
  const bool writes = (part & REST) == 0;
  const int t_begin = chunk * p.L, t_end = min(p.S, t_begin + p.L);     // this CTA's tokens of row b
  const int first = max(t_begin, (p.pad_left ? p.pad_left[b] : 0) - (p.cache_len ? *p.cache_len : 0));
  if (part == 0 && MODE != 1)
    for (int s = t_begin; s < min(first, t_end); ++s)
      for (int c = 0; c < GT_C; ++c)
        if (col0 + c < p.Dv) p.o[((size_t)(b * p.S + s) * p.H + h) * p.Dv + col0 + c] = 0.0f;
  // one thread copies: the records of a stage's tokens as they lie (a local scan leaves the queries out), two stages ahead of their use
  const int dvp = (p.Dv + 3) & ~3, vcol0 = blockIdx.x * cols;
  constexpr int Q0 = MODE == 1 ? P * GT_PITCH : 0;
  const uint32_t full = tc::smem_u32(bars);
  const float* row0 = rec + ((size_t)b * p.S * p.H + h) * RF;
  auto issue = [&](int s0, int stage) {
    const int nt = min(GS_TS, t_end - s0), nv = min(cols, dvp - vcol0);
    const uint32_t bar = full + 8u * stage;
    const float* src = row0 + (size_t)s0 * p.H * RF;
    uint32_t dst = tc::smem_u32(smem + (size_t)stage * GS_TS * SF);
    tc::mbar_expect_tx(bar, (uint32_t)(nt * (QKA - Q0 + nv) * 4));
    for (int t = 0; t < nt; ++t, src += (size_t)p.H * RF, dst += 4 * SF) {
      if (vcol0 == 0) {
        bulk_copy(dst + 4 * Q0, src + Q0, (QKA - Q0 + nv) * 4, bar);
      } else {
        bulk_copy(dst + 4 * Q0, src + Q0, (QKA - Q0) * 4, bar);
        bulk_copy(dst + 4 * QKA, src + QKA + vcol0, nv * 4, bar);
      }
    }
  };
  if (tid == 0) {
    tc::mbar_init(full, 1); tc::mbar_init(full + 8, 1);
    tc::fence_barrier_init();
    if (first < t_end) issue(first, 0);
    if (first + GS_TS < t_end) issue(first + GS_TS, 1);
  }
  __syncthreads();
  int stage = 0, phase = 0;
  for (int s0 = first; s0 < t_end; s0 += GS_TS) {
    tc::mbar_wait(full + 8u * stage, phase);
    const int nt = idle ? 0 : min(GS_TS, t_end - s0);
    const float* base = smem + (size_t)stage * GS_TS * SF;
    for (int t = 0; t < nt; ++t) {
      const float* tk = base + t * SF;
      unsigned long long v[GT_C];
      {
        const float4 vv = *reinterpret_cast<const float4*>(tk + QKA + grp * GT_C);
        v[0] = f2_dup(vv.x); v[1] = f2_dup(vv.y); v[2] = f2_dup(vv.z); v[3] = f2_dup(vv.w);
      }
      const ulonglong2* qt = reinterpret_cast<const ulonglong2*>(tk + part * GT_PITCH);
      const ulonglong2* kt = reinterpret_cast<const ulonglong2*>(tk + (P + part) * GT_PITCH);
      const ulonglong2* at = reinterpret_cast<const ulonglong2*>(tk + (2 * P + part) * GT_PITCH);
      unsigned long long acc[GT_C][2];
#pragma unroll
      for (int c = 0; c < GT_C; ++c) acc[c][0] = acc[c][1] = 0ull;       // (two zeros)
#pragma unroll
      for (int r = 0; r < GT_DP / 4; ++r) {
        const ulonglong2 al = at[r], kk = kt[r];
        ulonglong2 qq = make_ulonglong2(0ull, 0ull);
        if (MODE != 1) qq = qt[r];
        if (MODE == 1 && decays) { ap[2 * r] = f2_mul(ap[2 * r], al.x); ap[2 * r + 1] = f2_mul(ap[2 * r + 1], al.y); }
#pragma unroll
        for (int c = 0; c < GT_C; ++c) {
          st[2 * r][c] = f2_fma(al.x, st[2 * r][c], f2_mul(kk.x, v[c]));
          st[2 * r + 1][c] = f2_fma(al.y, st[2 * r + 1][c], f2_mul(kk.y, v[c]));
          if (MODE != 1) {
            acc[c][0] = f2_fma(qq.x, st[2 * r][c], acc[c][0]);
            acc[c][1] = f2_fma(qq.y, st[2 * r + 1][c], acc[c][1]);
          }
        }
      }
      if constexpr (MODE != 1) {                              // (a local scan leaves the read-outs to the second pass)
      float o[GT_C];
#pragma unroll
      for (int c = 0; c < GT_C; ++c) {
        const float2 x = f2_split(acc[c][0]), y = f2_split(acc[c][1]);
        o[c] = (x.x + x.y) + (y.x + y.y);
      }
      if constexpr (P >= 2) {                                 // keep two columns, give two
        const bool up = (part & (P / 2)) != 0;
        const float g0 = __shfl_xor_sync(0xffffffffu, up ? o[0] : o[2], P / 2), g1 = __shfl_xor_sync(0xffffffffu, up ? o[1] : o[3], P / 2);
        o[0] = (up ? o[2] : o[0]) + g0;
        o[1] = (up ? o[3] : o[1]) + g1;
      }
      if constexpr (P >= 4) {                                 // keep one, give one
        const bool up = (part & (P / 4)) != 0;
        const float g0 = __shfl_xor_sync(0xffffffffu, up ? o[0] : o[1], P / 4);
        o[0] = (up ? o[1] : o[0]) + g0;
#pragma unroll
        for (int off = P / 8; off > 0; off >>= 1) o[0] += __shfl_xor_sync(0xffffffffu, o[0], off);
      }
      if (writes) {
        float* dst = p.o + ((size_t)(b * p.S + s0 + t) * p.H + h) * p.Dv + ocol;
#pragma unroll
        for (int c = 0; c < NOUT; ++c) if (ocol + c < p.Dv) dst[c] = o[c];
      }
      }
    }
    __syncthreads();                                          // the stage is free
    if (tid == 0 && s0 + 2 * GS_TS < t_end) {
      fence_generic_to_bulk();                                // (its reads come before the copy that overwrites it)
      issue(s0 + 2 * GS_TS, stage);
    }
    stage ^= 1;
    phase ^= stage == 0;
  }
  if (MODE == 3) return;
#pragma unroll
  for (int r = 0; r < GT_DP / 2; ++r) {
    float2 x[GT_C];
#pragma unroll
    for (int c = 0; c < GT_C; ++c) x[c] = f2_split(st[r][c]);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int d = d0 + 2 * r + e;
      if (d >= p.D || col0 >= p.Dv) continue;
      float* dst = sbase + (size_t)d * p.Dv + col0;
      const float v[GT_C] = {e ? x[0].y : x[0].x, e ? x[1].y : x[1].x, e ? x[2].y : x[2].x, e ? x[3].y : x[3].x};
      if (vec) store4(dst, v);
      else
        for (int c = 0; c < GT_C; ++c) if (col0 + c < p.Dv) dst[c] = v[c];
    }
    if (decays && grp == 0) {
      const float2 a = f2_split(ap[r]);
      float* dst = p.cdecay + (((size_t)b * p.NC + chunk) * p.H + h) * p.D + d0 + 2 * r;
      if (d0 + 2 * r < p.D) dst[0] = a.x;
      if (d0 + 2 * r + 1 < p.D) dst[1] = a.y;
    }
  }
}

// Between the two passes: walk the chunks of a row in order.  cstate[c] holds the chunk's local end state on entry and the
// state the chunk starts from on exit; the row's state is advanced to the end of the prompt.
__global__ void gla_combine_kernel(GlaParams p) {
  pdl_wait();                      // programmatic dependent launch: nothing is read before the predecessor is done
  pdl_launch_dependents();
  const size_t per_row = (size_t)p.H * p.D * p.Dv, total = (size_t)p.B * per_row;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t b = i / per_row, e = i % per_row, hd = e / p.Dv;           // hd = h * D + d
    float s = p.state[i];
    for (int c0 = 0; c0 < p.NC; c0 += 8) {                    // eight chunks' loads in flight
      float local[8], dec[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int c = c0 + u;
        if (c >= p.NC) break;
        local[u] = p.cstate[((size_t)b * p.NC + c) * per_row + e];
        dec[u] = p.cdecay[((size_t)b * p.NC + c) * p.H * p.D + hd];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int c = c0 + u;
        if (c >= p.NC) break;
        p.cstate[((size_t)b * p.NC + c) * per_row + e] = s;
        s = fmaf(dec[u], s, local[u]);
      }
    }
    p.state[i] = s;
  }
}

}  // namespace jl

using namespace jl;

// Time chunks of a prompt scan.  A token costs some 250 cycles of dependent latency however few warps run, so while the grid is short
// of three CTAs per SM the prompt is cut into chunks that run side by side, in two passes (a local scan without read-outs, two thirds
// of the work, then the read-out pass) with a small kernel between them.  16 heads of 64 x 128, 2048 tokens of one row, both passes: 170 us in 10
// chunks, 143 in 20, 105 in 27 (one wave), 115 in 32.  (Projected decays and keys of up to 128 channels: gla_chunk.cu from 48 to 80 tokens on.)
static int gla_forced_chunks() {       // JLLAMA_GLA_CHUNKS: walks every prompt, in that many chunks where it has the tokens
  static const int forced = [] { const char* e = getenv("JLLAMA_GLA_CHUNKS"); return e ? atoi(e) : 0; }();
  return forced;
}
static int gla_chunks(int B, int S, int H, int D, int Dv) {
  const int forced = gla_forced_chunks();
  const int P = gla_lanes(D), threads = gla_threads(P, Dv), cols = threads / P * GT_C;
  const long warps = (long)B * H * ((Dv + cols - 1) / cols) * (threads / 32);
  int nc = (int)((long)SMS * 12 / (warps > 0 ? warps : 1));
  if (forced > 0) nc = forced;
  if (nc > S / 64) nc = S / 64;
  if (nc > 64) nc = 64;
  return nc < 2 ? 1 : nc;
}

extern "C" JL_API size_t jl_gla_scan_ws_floats(int B, int S, int H, int D, int Dv) {
  const int nc = gla_chunks(B, S, H, D, Dv);
  size_t n = (size_t)B * S * H * gla_record_floats(gla_lanes(D), Dv);
  if (nc > 1) n += (size_t)B * nc * H * D * Dv + (size_t)B * nc * H * D;
  if (gla_chunk_takes(B, S, H, D, Dv)) {                    // (one size for the calls that go to gla_chunk.cu and those that walk)
    const size_t chunked = gla_chunk_ws_floats(B, S, H, D, Dv);
    n = n > chunked ? n : chunked;
  }
  return n;
}

template <int P>
static int launch_stream(GlaParams p, float* ws, cudaStream_t st) {
  const int B = p.B, S = p.S, H = p.H, D = p.D, Dv = p.Dv;
  const int threads = gla_threads(P, Dv), cols = threads / P * GT_C;
  const size_t smem = (size_t)2 * GS_TS * (3 * P * GT_PITCH + cols) * sizeof(float);
  const int nc = gla_chunks(B, S, H, D, Dv);
  p.NC = nc;
  p.L = nc > 1 ? ((S + nc - 1) / nc + GS_TS - 1) / GS_TS * GS_TS : S;
  p.cstate = ws + (size_t)B * S * H * gla_record_floats(P, Dv);
  p.cdecay = p.cstate + (size_t)B * nc * H * D * Dv;
  const dim3 grid((Dv + cols - 1) / cols, H, B * nc), block(threads);
  if (smem > 48 * 1024) {
    JL_CUDA(cudaFuncSetAttribute(gla_stream_kernel<P, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    JL_CUDA(cudaFuncSetAttribute(gla_stream_kernel<P, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    JL_CUDA(cudaFuncSetAttribute(gla_stream_kernel<P, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  }
  if (nc == 1) {
    JL_LAUNCH_PDL((gla_stream_kernel<P, 0>), grid, block, smem, st, p, ws);
    JL_CUDA(cudaGetLastError());
    return JL_OK;
  }
  const size_t total = (size_t)B * H * D * Dv;
  JL_LAUNCH_PDL((gla_stream_kernel<P, 1>), grid, block, smem, st, p, ws);
  JL_CUDA(cudaGetLastError());
  JL_LAUNCH_PDL(gla_combine_kernel, dim3((unsigned)((total + 255) / 256 < 1184 ? (total + 255) / 256 : 1184)), dim3(256), 0, st, p);
  JL_CUDA(cudaGetLastError());
  JL_LAUNCH_PDL((gla_stream_kernel<P, 3>), grid, block, smem, st, p, ws);
  JL_CUDA(cudaGetLastError());
  return JL_OK;
}

// Both scans (projected decays; fixed decays with rotary q / k) share the kernels: what differs is in p.  walk: in fp32 FMAs token by token, whatever the sizes.
static int launch_scan(GlaParams p, const void* a2, const void* a2_bias, float* ws, int dtype, void* stream, bool walk = true) {
  const int B = p.B, S = p.S, H = p.H, D = p.D, Dv = p.Dv, R = p.R;
  int P = 1;
  while (P * GS_DP < D) P *= 2;
  JL_CHECK_ARG(P <= 32, "jl_gla_scan: key size %d above %d", D, 32 * GS_DP);
  const int cols = GS_THREADS / P;
  p.P = P;
  const size_t smem = (size_t)(3 * GS_TC * P * GS_PITCH + GS_TC * cols + GS_TC * R) * sizeof(float);
  JL_CHECK_ARG(smem <= 200 * 1024, "jl_gla_scan: key size %d with rank %d does not fit the staging buffer", D, R);
  dim3 grid((Dv + cols - 1) / cols, H, B), block(GS_THREADS);
  if (ws != nullptr && D <= GT_MAX_D) {                      // prompts: token-parallel preparation, then the pipe
    cudaStream_t st = (cudaStream_t)stream;
    if (!walk && gla_forced_chunks() <= 0 && gla_chunk_takes(B, S, H, D, Dv)) return gla_chunk_launch(p, a2, a2_bias, ws, dtype, st);
    p.P = gla_lanes(D);
    const int slots = H * (p.P * GT_DP + ((Dv + 3) & ~3));
    const dim3 pgrid((B * S + GP_TOK - 1) / GP_TOK, (slots + GP_THREADS - 1) / GP_THREADS);
    const size_t zsm = (size_t)GP_TOK * R * sizeof(float);     // (the check above leaves at most 200 KB)
    if (zsm > 48 * 1024)
      JL_DISPATCH_DTYPE(dtype, JL_CUDA(cudaFuncSetAttribute(gla_prep_kernel<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)zsm)));
    if (gla_plain(p, a2, dtype == DT_BF16 ? 2 : 4))
      JL_DISPATCH_DTYPE(dtype, JL_LAUNCH_PDL((gla_prep_kernel<T, true>), pgrid, dim3(GP_THREADS), zsm, st, p, (const T*)a2, (const T*)a2_bias, ws));
    else
      JL_DISPATCH_DTYPE(dtype, JL_LAUNCH_PDL((gla_prep_kernel<T, false>), pgrid, dim3(GP_THREADS), zsm, st, p, (const T*)a2, (const T*)a2_bias, ws));
    JL_CUDA(cudaGetLastError());
    switch (p.P) {
      case 1: return launch_stream<1>(p, ws, st);
      case 2: return launch_stream<2>(p, ws, st);
      case 4: return launch_stream<4>(p, ws, st);
      case 8: return launch_stream<8>(p, ws, st);
      default: return launch_stream<16>(p, ws, st);
    }
  }
  if (smem > 48 * 1024) {
    if (dtype == DT_BF16) JL_CUDA(cudaFuncSetAttribute(gla_scan_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    else JL_CUDA(cudaFuncSetAttribute(gla_scan_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  }
  JL_DISPATCH_DTYPE(dtype, JL_LAUNCH_PDL(gla_scan_kernel<T>, dim3(grid), dim3(block), smem, (cudaStream_t)stream, p, (const T*)a2, (const T*)a2_bias));
  JL_CUDA(cudaGetLastError());
  return JL_OK;
}

static int gla_scan(const float* y, int ldy, int q_off, int k_off, int v_off, int a_off, const void* a2, const void* a2_bias, float* state, float* o,
                    const int* cache_len, const int* pad_left, int B, int S, int H, int D, int Dv, int R, float q_scale, float tau, float* ws, int dtype,
                    void* stream, bool walk) {
  JL_CHECK_ARG(B >= 1 && S >= 1 && H >= 1 && D >= 1 && Dv >= 1 && R >= 1, "jl_gla_scan: bad shape");
  JL_CHECK_ARG(tau > 0.0f, "jl_gla_scan: tau=%f must be positive", tau);
  GlaParams p{y, ldy, q_off, k_off, v_off, a_off, B, S, H, D, Dv, R, 1, q_scale, 1.0f / tau, cache_len, pad_left, state, o};
  p.k_scale = 1.0f;
  return launch_scan(p, a2, a2_bias, ws, dtype, stream, walk);
}

extern "C" JL_API int jl_gla_scan(const float* y, int ldy, int q_off, int k_off, int v_off, int a_off, const void* a2,
                                  const void* a2_bias, float* state, float* o, const int* cache_len, const int* pad_left, int B,
                                  int S, int H, int D, int Dv, int R, float q_scale, float tau, float* ws, int dtype,
                                  void* stream) {
  return gla_scan(y, ldy, q_off, k_off, v_off, a_off, a2, a2_bias, state, o, cache_len, pad_left, B, S, H, D, Dv, R, q_scale, tau, ws, dtype, stream, false);
}

extern "C" JL_API int jl_gla_scan_exact(const float* y, int ldy, int q_off, int k_off, int v_off, int a_off, const void* a2,
                                        const void* a2_bias, float* state, float* o, const int* cache_len, const int* pad_left, int B,
                                        int S, int H, int D, int Dv, int R, float q_scale, float tau, float* ws, int dtype,
                                        void* stream) {
  return gla_scan(y, ldy, q_off, k_off, v_off, a_off, a2, a2_bias, state, o, cache_len, pad_left, B, S, H, D, Dv, R, q_scale, tau, ws, dtype, stream, true);
}

extern "C" JL_API int jl_retention_scan(const float* y, int ldy, int q_off, int k_off, int v_off, const float* head_decay,
                                        const float* cos_t, const float* sin_t, int max_pos, int rot, int layout, float q_scale,
                                        float k_scale, float* state, float* o, const int* cache_len, const int* pad_left, int B,
                                        int S, int H, int D, int Dv, float* ws, void* stream) {
  JL_CHECK_ARG(B >= 1 && S >= 1 && H >= 1 && D >= 1 && Dv >= 1 && head_decay != nullptr, "jl_retention_scan: bad shape");
  JL_CHECK_ARG(rot >= 0 && rot <= D && rot % 2 == 0 && (layout == 0 || layout == 1), "jl_retention_scan: rot=%d of D=%d, layout %d",
               rot, D, layout);
  GlaParams p{y, ldy, q_off, k_off, v_off, 0, B, S, H, D, Dv, 0, 1, q_scale, 1.0f, cache_len, pad_left, state, o};
  p.head_decay = head_decay; p.cos_t = cos_t; p.sin_t = sin_t; p.rot = rot; p.layout = layout; p.max_pos = max_pos;
  p.k_scale = k_scale;
  return launch_scan(p, nullptr, nullptr, ws, DT_F32, stream);
}

extern "C" JL_API int jl_ssd_scan(const float* u, int ldu, int q_off, int k_off, int v_off, int G, const float* aux, float* state,
                                  float* o, const int* cache_len, const int* pad_left, int B, int S, int H, int D, int Dv,
                                  float* ws, void* stream) {
  JL_CHECK_ARG(B >= 1 && S >= 1 && H >= 1 && D >= 1 && Dv >= 1 && aux != nullptr, "jl_ssd_scan: bad shape");
  JL_CHECK_ARG(G >= 1 && H % G == 0, "jl_ssd_scan: %d heads in %d groups", H, G);
  GlaParams p{u, ldu, q_off, k_off, v_off, 0, B, S, H, D, Dv, 0, 1, 1.0f, 1.0f, cache_len, pad_left, state, o};
  p.k_scale = 1.0f;
  p.qk_div = H / G; p.aux = aux; p.ld_aux = 2 * H;
  return launch_scan(p, nullptr, nullptr, ws, DT_F32, stream);
}

// One fixed decay per head over projections that pass an activation (no rotation, no scale): S_t = decay_h S_(t-1) + k_t v_t^T.
extern "C" JL_API int jl_activated_scan(const float* y, int ldy, int q_off, int k_off, int v_off, const float* head_decay, int act,
                                        float* state, float* o, const int* cache_len, const int* pad_left, int B, int S, int H, int D,
                                        int Dv, float* ws, void* stream) {
  JL_CHECK_ARG(B >= 1 && S >= 1 && H >= 1 && D >= 1 && Dv >= 1 && head_decay != nullptr, "jl_activated_scan: bad shape");
  JL_CHECK_ARG(act == ACT_NONE || act == ACT_SILU || act == ACT_SIGMOID || act == ACT_GELU_TANH || act == ACT_RELU2,
               "jl_activated_scan: activation %d", act);
  GlaParams p{y, ldy, q_off, k_off, v_off, 0, B, S, H, D, Dv, 0, 1, 1.0f, 1.0f, cache_len, pad_left, state, o};
  p.head_decay = head_decay; p.k_scale = 1.0f; p.act = act;
  return launch_scan(p, nullptr, nullptr, ws, DT_F32, stream);
}

// Matrix memory: decay and value scale per (token, head) from aux [M][ld_aux] (columns h and H + h), Dv value columns of y followed by
// one column of ones; state [B][H][D][Dv + 1], o [M][H][Dv + 1] (last column: n . q).  ws as for Dv + 1 columns.
extern "C" JL_API int jl_mlstm_scan(const float* y, int ldy, int q_off, int k_off, int v_off, const float* aux, int ld_aux, float q_scale,
                                    float* state, float* o, const int* cache_len, const int* pad_left, int B, int S, int H, int D,
                                    int Dv, float* ws, void* stream) {
  JL_CHECK_ARG(B >= 1 && S >= 1 && H >= 1 && D >= 1 && Dv >= 1 && aux != nullptr && ld_aux >= 2 * H, "jl_mlstm_scan: bad shape");
  GlaParams p{y, ldy, q_off, k_off, v_off, 0, B, S, H, D, Dv + 1, 0, 1, q_scale, 1.0f, cache_len, pad_left, state, o};
  p.k_scale = 1.0f; p.aux = aux; p.ld_aux = ld_aux; p.ones = 1;
  return launch_scan(p, nullptr, nullptr, ws, DT_F32, stream);
}

// One token per row of the scan with projected decays, then the norm of every head's read-out (weight norm [Dv] or nullptr) and the gate
// act(y[:, g_off + ...]): out [B, H * Dv] of dtype.  JL_ERR_UNSUPPORTED: sizes whose heads do not fit a CTA (the two launches take them).
extern "C" JL_API int jl_gla_step(const float* y, int ldy, int q_off, int k_off, int v_off, int a_off, int g_off, const void* a2, const void* a2_bias,
                                  const void* norm, float* state, void* out, const int* cache_len, const int* pad_left, int B, int H, int D, int Dv,
                                  int R, float q_scale, float tau, float eps, int gate_act, int dtype, void* stream) {
  JL_CHECK_ARG(B >= 1 && H >= 1 && D >= 1 && Dv >= 1 && R >= 1, "jl_gla_step: bad shape");
  JL_CHECK_ARG(tau > 0.0f, "jl_gla_step: tau=%f must be positive", tau);
  JL_CHECK_ARG(gate_act >= 0 && gate_act <= ACT_LAST, "jl_gla_step: bad activation %d", gate_act);
  const int cols = (Dv + 31) & ~31;
  // 16 channels a thread where that is at most 512 threads (more loads in flight than 32; above, 32 keep the CTA small)
  const int dp = cols * ((D + 15) / 16) <= 512 ? 16 : 32, threads = cols * ((D + dp - 1) / dp);
  if (threads > 1024 || B > 65535) return JL_ERR_UNSUPPORTED;
  GlaStep s{GlaParams{y, ldy, q_off, k_off, v_off, a_off, B, 1, H, D, Dv, R, 1, q_scale, 1.0f / tau, cache_len, pad_left, state, nullptr}, g_off, eps, gate_act};
  s.p.k_scale = 1.0f;
  size_t smem = (size_t)(3 * threads / cols * dp + threads) * sizeof(float);             // (16 KB at most)
  if ((long)H * B <= SMS) {
    // placed while the projection before fills most SMs, the CTAs came to lie many to an SM: with this much each has its own (us in a graph, a layer of 3 rows x 16 heads of 16 x 64
    // 12.0 -> 11.1, 7 x 8 heads of 100 x 128 18.6 -> 17.3; in two launches 11.3 and 19.7)
    smem = 116 * 1024;
    if (dp == 16) JL_DISPATCH_DTYPE(dtype, JL_CUDA(cudaFuncSetAttribute((gla_step_kernel<T, 16>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)));
    else JL_DISPATCH_DTYPE(dtype, JL_CUDA(cudaFuncSetAttribute((gla_step_kernel<T, 32>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)));
  }
  if (dp == 16)
    JL_DISPATCH_DTYPE(dtype, JL_LAUNCH_PDL((gla_step_kernel<T, 16>), dim3(H, B), dim3(threads), smem, (cudaStream_t)stream, s, (const T*)a2,
                                           (const T*)a2_bias, (const T*)norm, (T*)out));
  else
    JL_DISPATCH_DTYPE(dtype, JL_LAUNCH_PDL((gla_step_kernel<T, 32>), dim3(H, B), dim3(threads), smem, (cudaStream_t)stream, s, (const T*)a2,
                                           (const T*)a2_bias, (const T*)norm, (T*)out));
  JL_CUDA(cudaGetLastError());
  return JL_OK;
}

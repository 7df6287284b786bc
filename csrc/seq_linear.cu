// Linear layers for any shape and for bfloat16 or true float32 operands: y = act(x W^T) with W [N, K] (out, in).
//
//  * linear_mma_rows_kernel (bfloat16, M = 3 .. 8: decode) — weight-streaming through mma.sync: see there.
//  * linear_flow_kernel  (bfloat16, M <= 4) — the sums of the next one by CTAs that stay: see there.
//  * linear_rows_kernel  (M <= 8: float32, pitches without 16-byte rows) — weight-streaming: a CTA owns ROWS output features, its 8 warps split K, each
//    lane reads 16 bytes of every row per step (all loads issued before the first use) and keeps ROWS x M fp32
//    accumulators; activations come from L1; the warps' sums meet in shared memory in a fixed order.
//  * linear_f32_kernel   (float32, M > 8, linear_f32.cu) — tensor cores with the accuracy of fp32 FMAs.
//  * linear_tiled_kernel (any M)           — 64 x 64 x 16 shared-memory tiles, 4 x 4 outputs per thread, fp32 FMA: the fall-back
//    for sizes, pitches and addresses that the tensor-core kernels do not take.
//
// Products and sums are fp32 (or as good: linear_f32.cu), never TF32.  The output is fp32 or the operand type, written at a column offset
// of a wider row (ldo) so that projections that share an input can share an output buffer.
#include "jllama_b200.h"
#include "linear_f32.cuh"
#include "seq_types.cuh"

namespace jl {

constexpr int LR_ROWS = 4;      // output features per warp
constexpr int LR_MAXM = 8;

template <typename T> struct Vec;                    // 16-byte vector of T
template <> struct Vec<float> { static constexpr int N = 4; };
template <> struct Vec<__nv_bfloat16> { static constexpr int N = 8; };

template <typename T> __device__ __forceinline__ void load_vec(const T* p, float (&v)[Vec<T>::N]);
template <> __device__ __forceinline__ void load_vec<float>(const float* p, float (&v)[4]) {
  float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
template <> __device__ __forceinline__ void load_vec<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[8]) {
  uint4 t = *reinterpret_cast<const uint4*>(p);
  v[0] = bf16_lo(t.x); v[1] = bf16_hi(t.x); v[2] = bf16_lo(t.y); v[3] = bf16_hi(t.y);
  v[4] = bf16_lo(t.z); v[5] = bf16_hi(t.z); v[6] = bf16_lo(t.w); v[7] = bf16_hi(t.w);
}

__device__ __forceinline__ void unpack8(const uint4& t, float (&v)[8]) {
  v[0] = bf16_lo(t.x); v[1] = bf16_hi(t.x); v[2] = bf16_lo(t.y); v[3] = bf16_hi(t.y);
  v[4] = bf16_lo(t.z); v[5] = bf16_hi(t.z); v[6] = bf16_lo(t.w); v[7] = bf16_hi(t.w);
}
__device__ __forceinline__ uint4 ldg_weights(const void* p) {     // touched once: no line in L1 (the tokens live there)
  uint4 r;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p) : "memory");
  return r;
}

constexpr int LR_WARPS = 8;     // warps of a CTA: they split K for the same LR_ROWS output features

template <typename T, typename OutT, int M>
__global__ void __launch_bounds__(LR_WARPS * 32) linear_rows_kernel(const T* __restrict__ x, int ldx, const T* __restrict__ w,
                                                                    OutT* __restrict__ out, int ldo, int N, int K, int act,
                                                                    float p0, float p1, int vec_ok, LinearGroup g) {
  pdl_wait();                      // programmatic dependent launch: nothing is read before the predecessor is done
  pdl_launch_dependents();
  __shared__ float red[LR_WARPS][LR_ROWS][M];
  if (g.w_index && g.w_index[blockIdx.y] < 0) return;            // a batch without a matrix (uniform for the CTA): nothing is written
  {
    const long long z = blockIdx.y;
    x += (z / g.x_div) * g.x_bs;
    w += (g.w_index ? (long long)g.w_index[z] : z) * g.w_bs;
    out += z * g.o_bs;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n0 = blockIdx.x * LR_ROWS;
  float acc[LR_ROWS][M];
#pragma unroll
  for (int r = 0; r < LR_ROWS; ++r)
#pragma unroll
    for (int m = 0; m < M; ++m) acc[r][m] = 0.0f;
  constexpr int VN = Vec<T>::N;
  int k_done = 0;
  if (vec_ok) {
    const int kv = K / VN * VN;
    for (int k = (warp * 32 + lane) * VN; k < kv; k += LR_WARPS * 32 * VN) {
      float wv[LR_ROWS][VN];
#pragma unroll
      for (int r = 0; r < LR_ROWS; ++r) {          // all weight loads of this step are in flight before any is used
        const int n = min(n0 + r, N - 1);
        load_vec<T>(w + (size_t)n * K + k, wv[r]);
      }
#pragma unroll
      for (int m = 0; m < M; ++m) {
        float xv[VN];
        load_vec<T>(x + (size_t)m * ldx + k, xv);
#pragma unroll
        for (int r = 0; r < LR_ROWS; ++r)
#pragma unroll
          for (int j = 0; j < VN; ++j) acc[r][m] = fmaf(wv[r][j], xv[j], acc[r][m]);
      }
    }
    k_done = kv;
  }
  for (int k = k_done + warp * 32 + lane; k < K; k += LR_WARPS * 32) {
#pragma unroll
    for (int r = 0; r < LR_ROWS; ++r) {
      const float wv = to_f(w[(size_t)min(n0 + r, N - 1) * K + k]);
#pragma unroll
      for (int m = 0; m < M; ++m) acc[r][m] = fmaf(wv, to_f(x[(size_t)m * ldx + k]), acc[r][m]);
    }
  }
#pragma unroll
  for (int r = 0; r < LR_ROWS; ++r)
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const float s = warp_sum(acc[r][m]);
      if (lane == 0) red[warp][r][m] = s;
    }
  __syncthreads();
  if (threadIdx.x < LR_ROWS * M) {
    const int r = threadIdx.x / M, m = threadIdx.x % M;
    float s = 0.0f;
#pragma unroll
    for (int wq = 0; wq < LR_WARPS; ++wq) s += red[wq][r][m];
    if (n0 + r < N) out[(size_t)m * ldo + n0 + r] = from_f<OutT>(apply_act(s, act, p0, p1));
  }
}

// bfloat16, up to 4 tokens, one matrix: the same sums in the same order, but the CTAs stay (FL_CTAS per SM) and walk the groups of four output
// features, the next group's (or next 2048 k's) weights already on their way into registers while this one is multiplied; and where the
// weights are known to be a parameter the first ones are requested BEFORE the wait for the kernels ahead.  Bound: the weights' way from
// memory; a CTA per group spends itself on coming and going where K is short (one load round each).
// One B200, us in a chain of cold weights, linear_rows_kernel -> this -> this with the early request (features x K): 1 token 2048 x 2048 3.9 -> 3.4 ->
// 2.4, 8192 x 2048 9.1 -> 8.6 -> 7.6, 32000 x 2048 27.4 -> 26.1 -> 25.0, 2048 x 8192 8.7 -> 7.8 -> 6.9, 4096 x 14336 24.9 -> 22.1 -> 21.2 (5.5 TB/s).
// 3 and 4 tokens: what linear_mma_rows_kernel leaves (4 tokens 2048 x 2048 5.8 -> 5.4 -> 4.2, 2048 x 1024 4.6 -> 4.4 -> 3.6).  Where it is not taken: flow_takes.
constexpr int fl_ctas(int m) { return m <= 2 ? 4 : 3; }          // per SM

template <typename OutT, int M>
__global__ void __launch_bounds__(LR_WARPS * 32, fl_ctas(M)) linear_flow_kernel(const __nv_bfloat16* __restrict__ x, int ldx,
                                                                    const __nv_bfloat16* __restrict__ w, OutT* __restrict__ out, int ldo,
                                                                    int N, int K, int act, float p0, float p1, int early) {
  constexpr int NV = M == 3 ? 16 : 4 * M, STEP = LR_WARPS * 32 * 8;       // sums of a thread, to a power of two; k of a round
  __shared__ float red[2][LR_WARPS][NV];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = (N + LR_ROWS - 1) / LR_ROWS, steps = (K + STEP - 1) / STEP;
  int g = blockIdx.x, s = 0;                               // the round that is loaded
  uint4 wv[LR_ROWS];
  auto load = [&](int gl, int sl) {
    const int k = sl * STEP + (int)threadIdx.x * 8;
    const __nv_bfloat16* row = w + (size_t)gl * LR_ROWS * K + k;
#pragma unroll
    for (int r = 0; r < LR_ROWS; ++r)
      wv[r] = k < K && gl < groups ? ldg_weights(row + (size_t)min(r, N - 1 - gl * LR_ROWS) * K) : make_uint4(0u, 0u, 0u, 0u);
  };
  if (early) load(g, 0);
  pdl_wait();
  pdl_launch_dependents();
  if (!early) load(g, 0);
  float acc[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) acc[i] = 0.0f;
  int buf = 0;
  while (g < groups) {
    const int k = s * STEP + (int)threadIdx.x * 8;
    uint4 xv[M];
#pragma unroll
    for (int m = 0; m < M; ++m) xv[m] = k < K ? *reinterpret_cast<const uint4*>(x + (size_t)m * ldx + k) : make_uint4(0u, 0u, 0u, 0u);
    float wf[LR_ROWS][8];
#pragma unroll
    for (int r = 0; r < LR_ROWS; ++r) unpack8(wv[r], wf[r]);
    const int g0 = g;
    const bool last = s + 1 == steps;
    s = last ? 0 : s + 1;
    if (last) g += gridDim.x;
    load(g, s);                                            // in flight during everything below
    if (k < K) {
#pragma unroll
      for (int m = 0; m < M; ++m) {
        float xf[8];
        unpack8(xv[m], xf);
#pragma unroll
        for (int r = 0; r < LR_ROWS; ++r)
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[r * M + m] = fmaf(wf[r][j], xf[j], acc[r * M + m]);
      }
    }
    if (last) {
      // fold: at each step a lane keeps half of its sums and gives the other half to its partner (the additions of warp_sum)
      int idx = 0;
#pragma unroll
      for (int o = 16, n = NV; o > 0; o >>= 1) {
        if (n > 1) {
          const bool up = (lane & o) != 0;
          n >>= 1;
          idx = idx * 2 + (up ? 1 : 0);
#pragma unroll
          for (int i = 0; i < NV / 2; ++i)
            if (i < n) {
              const float keep = up ? acc[i + n] : acc[i], give = up ? acc[i] : acc[i + n];
              acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        } else {
          acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
        }
      }
      if ((lane & (32 / NV - 1)) == 0) red[buf][warp][idx] = acc[0];
      __syncthreads();                                     // (a buffer is written again only after the next one of these)
      if (threadIdx.x < LR_ROWS * M) {
        const int r = threadIdx.x / M, m = threadIdx.x % M;
        float t = 0.0f;
#pragma unroll
        for (int wq = 0; wq < LR_WARPS; ++wq) t += red[buf][wq][threadIdx.x];
        if (g0 * LR_ROWS + r < N) out[(size_t)m * ldo + g0 * LR_ROWS + r] = from_f<OutT>(apply_act(t, act, p0, p1));
      }
      buf ^= 1;
#pragma unroll
      for (int i = 0; i < NV; ++i) acc[i] = 0.0f;
    }
  }
}

// Where linear_flow_kernel is the faster of the two (the same bits).  What it gains it loses again where the last of its rounds is a short one, and with two tokens
// more CTAs hide a round better than its few.  us, linear_rows_kernel | this | this with the early request (tokens: features x K):
//   1: 3000 x 2048 4.3 | 4.6 | 3.4, 3000 x 4096 6.3 | 7.4 | 6.4, 3000 x 8192 10.4 | 12.9 | 11.8 (a quarter of the second round), 8192 x 3072 12.5 | 12.9 | 11.8;
//   2: 2048 x 2048 3.7 | 3.9 | 2.7, 8192 x 2048 9.8 | 10.5 | 9.2, 16384 x 2048 17.4 | 17.0 | 15.8, 2048 x 4096 5.1 | 5.7 | 4.7, 8192 x 4096 15.1 | 17.2 | 16.1;
//   4: 2048 x 4096 8.1 | 8.5 | 7.2, 2048 x 2048 5.6 | 5.3 | 4.1.
static bool flow_takes(int M, int N, int K, bool early) {
  const int groups = (N + LR_ROWS - 1) / LR_ROWS, most = SMS * fl_ctas(M);
  if (M == 1) {
    if (groups > most && 2 * groups <= 3 * most) return early && K <= 3072;
    return early || groups <= 2 * most || K <= 2048;
  }
  if (M == 2) return early ? K <= 2048 || (groups <= most && K <= 4096) : groups >= 5 * most && K <= 2048;
  return M <= 4 && K <= (M == 3 || early ? 4096 : 2048);
}

template <typename OutT>
static int flow_launch(const __nv_bfloat16* x, int ldx, const __nv_bfloat16* w, OutT* out, int ldo, int M, int N, int K, int act, float p0,
                       float p1, bool early, cudaStream_t st) {
  const int groups = (N + LR_ROWS - 1) / LR_ROWS;
#define JL_FL(MM)                                                                                                        \
  case MM: {                                                                                                             \
    const int most = SMS * fl_ctas(MM);                                                                          \
    JL_LAUNCH_PDL((linear_flow_kernel<OutT, MM>), dim3(groups < most ? groups : most), dim3(LR_WARPS * 32), 0, st, x, ldx, w, out, ldo, N, K, act, \
                  p0, p1, early ? 1 : 0);                                                                                \
    break;                                                                                                               \
  }
  switch (M) { JL_FL(1) JL_FL(2) JL_FL(3) JL_FL(4) }
#undef JL_FL
  return cudaGetLastError() == cudaSuccess ? JL_OK : JL_ERR_CUDA;
}

// bfloat16 weights of a decode step of 3 to 8 tokens, streamed once, tokens as the 8 columns of mma.sync.m16n8k16 (products exact,
// fp32 sums).  A warp takes 16 output features and one of KS parts of K in batches of 256 k: lane (g = lane / 4, t = lane % 4) loads the
// 16-byte chunks t, t + 4, ... of rows g and g + 8 straight into A fragments, and the same chunks of token g into B fragments (the order of
// k inside a product is free as long as both agree: MMA v of chunk u uses words 2v, 2v + 1), so a batch is 16 weight loads in flight
// per lane, 8 token loads (L1) and 16 MMAs.  The FMA kernel is bound by issue there: it unpacks every weight and multiplies it once per token.
// The tensor core truncates when it adds, so every MMA (16 k) starts from zero and its sums meet the rest in rounded fp32 additions; the KS
// warps of a CTA meet in shared memory, neighbours first.  Error against float64 (2-norm; features x K), FMA kernel -> this one, normal
// operands | of one sign: 2048 x 1536 7.4e-8 -> 7.2e-8 | 4.6e-8 -> 3.9e-8, 2048 x 2048 7.9e-8 -> 7.5e-8 | 4.8e-8 -> 4.4e-8, 8192 x 11008 9.3e-8 ->
// 9.0e-8 | 5.4e-8 -> 4.4e-8.  It is kept where it is the more exact one: from LM_MIN_K on (2048 x 1024: 6.8e-8 -> 7.0e-8 | 4.3e-8 -> 4.4e-8), and
// with at most LM_MAX_SEG k to a warp, whose batches are added one after the other (32000 features in parts of 2048 k 8.4e-8 -> 8.5e-8, of 4096 8.9e-8
// -> 10.0e-8).  (Chains of two MMAs: 5 % faster, but 5.4e-8 with operands of one sign at 2048 x 2048.)
// 8 tokens on one B200, FMA kernel -> this one (features x K; cold L2, launch included): 32000 x 2048 90 -> 37 us, 8192 x 2048 29.5 -> 18.4,
// 2048 x 8192 22.6 -> 18.3, 2048 x 2048 14.2 -> 10.1; 4 tokens, in a chain of cold weights: 32000 x 2048 50 -> 26.5, 28672 x 4096 65 -> 44, 8192 x 2048 14.6 -> 10.7,
// 2048 x 8192 12.8 -> 10.6, 6160 x 2048 11.7 -> 6.8 (3 tokens: 42.5, 57.8, 12.9, 12.9, 10.4 before).  With 1 or 2 tokens the FMA kernels, whose loads run along a row (512
// contiguous bytes against 64), are as fast or faster (2 tokens: 2048 x 8192 7.9 against 10.5), and with fewer than 96 groups of 16 features too (8 tokens, 1024 x 5464:
// 7.4 against 8.9: a warp's batches run one after the other), with 3 or 4 tokens 192 (2048 x 2048: linear_flow_kernel, its weights asked for early, 4.2 against
// 4.6; 4096 x 2048: 7.0 against 5.9).
constexpr int LM_U = 8, LM_BATCH = 32 * LM_U;        // chunk groups of 32 k in flight; k of a batch
constexpr int LM_MIN_K = 1536, LM_MAX_SEG = 1536;

__device__ __forceinline__ void lm_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <typename OutT, int KS>
__global__ void __launch_bounds__((KS > 4 ? KS : 4) * 32) linear_mma_rows_kernel(const __nv_bfloat16* __restrict__ x, int ldx,
                                                                                 const __nv_bfloat16* __restrict__ w, OutT* __restrict__ out,
                                                                                 int ldo, int M, int N, int K, int act, float p0, float p1,
                                                                                 LinearGroup gr) {
  constexpr int WARPS = KS > 4 ? KS : 4, GROUPS = WARPS / KS;
  __shared__ float red[WARPS][16][9];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int part = warp % KS, n0 = (blockIdx.x * GROUPS + warp / KS) * 16;
  const int seg = ((K + KS - 1) / KS + 31) / 32 * 32;
  const int k0 = part * seg, k1 = min(K, k0 + seg);
  const long long z = blockIdx.y;
  pdl_wait();                      // programmatic dependent launch: nothing is read before the predecessor is done
  pdl_launch_dependents();
  if (gr.w_index && gr.w_index[z] < 0) return;             // a batch without a matrix (uniform for the CTA): nothing is written
  w += (gr.w_index ? (long long)gr.w_index[z] : z) * gr.w_bs;
  x += (z / gr.x_div) * gr.x_bs;
  out += z * gr.o_bs;
  float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  const __nv_bfloat16* w0 = w + (size_t)min(n0 + g, N - 1) * K;
  const __nv_bfloat16* w1 = w + (size_t)min(n0 + g + 8, N - 1) * K;
  const __nv_bfloat16* xr = x + (size_t)min(g, M - 1) * ldx;
  const bool tok = g < M;
  if (n0 < N) {
    for (int kb = k0; kb < k1; kb += LM_BATCH) {
      uint4 a[LM_U], b[LM_U], c[LM_U];
#pragma unroll
      for (int u = 0; u < LM_U; ++u) {                     // all loads of the batch before the first use
        const int k = kb + 32 * u + 8 * t;
        const bool on = k < k1;                            // K is a multiple of 8
        a[u] = on ? ldg_weights(w0 + k) : make_uint4(0u, 0u, 0u, 0u);
        b[u] = on ? ldg_weights(w1 + k) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < LM_U; ++u) {
        const int k = kb + 32 * u + 8 * t;
        c[u] = tok && k < k1 ? *reinterpret_cast<const uint4*>(xr + k) : make_uint4(0u, 0u, 0u, 0u);
      }
      float d[LM_U][4];
#pragma unroll
      for (int u = 0; u < LM_U; ++u) {
        float e[2][4] = {};
        lm_mma(e[0], a[u].x, b[u].x, a[u].y, b[u].y, c[u].x, c[u].y);
        lm_mma(e[1], a[u].z, b[u].z, a[u].w, b[u].w, c[u].z, c[u].w);
#pragma unroll
        for (int i = 0; i < 4; ++i) d[u][i] = e[0][i] + e[1][i];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        sum[i] += ((d[0][i] + d[1][i]) + (d[2][i] + d[3][i])) + ((d[4][i] + d[5][i]) + (d[6][i] + d[7][i]));
    }
  }
  red[warp][g][2 * t] = sum[0]; red[warp][g][2 * t + 1] = sum[1];
  red[warp][g + 8][2 * t] = sum[2]; red[warp][g + 8][2 * t + 1] = sum[3];
  __syncthreads();
  for (int i = threadIdx.x; i < GROUPS * 16 * M; i += WARPS * 32) {
    const int gi = i / (16 * M), m = i / 16 % M, r = i % 16;
    float s[KS];
#pragma unroll
    for (int q = 0; q < KS; ++q) s[q] = red[gi * KS + q][r][m];
#pragma unroll
    for (int o = 1; o < KS; o <<= 1)
#pragma unroll
      for (int q = 0; q < KS; q += 2 * o) s[q] += s[q + o];          // neighbouring parts first
    const int n = (blockIdx.x * GROUPS + gi) * 16 + r;
    if (n < N) out[(size_t)m * ldo + n] = from_f<OutT>(apply_act(s[0], act, p0, p1));
  }
}

static int lm_parts(long groups, int K) {
  int ks = 1;
  while (ks < 16 && (K > ks * LM_MAX_SEG || (groups * ks < SMS * 14 && K >= 2 * ks * (LM_BATCH / 2)))) ks *= 2;
  return ks;
}
// Long K whose CTAs (8 parts: three to an SM) need a second round for a quarter of them or less: with 3 or 4 tokens linear_rows_kernel is the faster there
// (3 tokens, 8192 x 8192 31.1 against 34.8 us; 4096 x 8192 18.9 against 13.8, 12288 x 8192 44.1 against 39.8).
static bool lm_short_tail(int N, int K, int nbatch) {
  const long groups = (long)((N + 15) / 16) * nbatch, slots = SMS * 3;
  return K > 4096 && lm_parts(groups, K) == 8 && groups > slots && 4 * groups <= 5 * slots;
}

template <typename OutT>
static void lm_launch(const __nv_bfloat16* x, int ldx, const __nv_bfloat16* w, OutT* out, int ldo, int M, int N, int K, int act, float p0,
                      float p1, cudaStream_t st, const LinearGroup& g, int nbatch) {
  // parts of K: some 14 warps on every SM (8 KB in flight each), each part at least half a batch long, at most LM_MAX_SEG
  const long groups = (long)((N + 15) / 16) * nbatch;
  const int ks = lm_parts(groups, K);
  const int per = (ks > 4 ? 1 : 4 / ks) * 16;
  const dim3 grid((N + per - 1) / per, nbatch), block((ks > 4 ? ks : 4) * 32);
#define JL_LM(KS_) case KS_: JL_LAUNCH_PDL((linear_mma_rows_kernel<OutT, KS_>), grid, block, 0, st, x, ldx, w, out, ldo, M, N, K, act, p0, p1, g); break;
  switch (ks) { JL_LM(1) JL_LM(2) JL_LM(4) JL_LM(8) JL_LM(16) }
#undef JL_LM
}

constexpr int LT_BN = 64, LT_BK = 16;              // (LT_BM rows: linear_f32.cuh)

template <typename T, typename OutT>
__global__ void __launch_bounds__(256) linear_tiled_kernel(const T* __restrict__ x, int ldx, const T* __restrict__ w,
                                                           OutT* __restrict__ out, int ldo, int M, int N, int K, int act,
                                                           float p0, float p1, LinearGroup g) {
  pdl_wait();                      // programmatic dependent launch: nothing is read before the predecessor is done
  pdl_launch_dependents();
  __shared__ float xs[LT_BK][LT_BM + 4];
  __shared__ float ws[LT_BK][LT_BN + 4];
  __shared__ int srow[LT_BM];
  const int m0 = blockIdx.y * LT_BM, n0 = blockIdx.x * LT_BN;
  if (g.tile_group) {
    const int e = g.tile_group[blockIdx.y];
    if (e < 0) return;                                             // uniform for the CTA
    w += (long long)e * g.w_bs;
  } else {
    const long long z = blockIdx.z;
    if (g.w_index && g.w_index[z] < 0) return;                     // a batch without a matrix (uniform for the CTA)
    x += (z / g.x_div) * g.x_bs;
    w += (g.w_index ? (long long)g.w_index[z] : z) * g.w_bs;
    out += z * g.o_bs;
  }
  if (threadIdx.x < LT_BM) {
    const int gm = m0 + threadIdx.x;
    srow[threadIdx.x] = gm < M ? ((g.tile_group && g.row_src) ? g.row_src[gm] : gm) : -1;
  }
  __syncthreads();
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;         // 16 x 16 threads, 4 x 4 outputs each
  float acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += LT_BK) {
    for (int i = threadIdx.x; i < LT_BM * LT_BK; i += 256) {
      const int r = i / LT_BK, c = i % LT_BK;
      const int gn = n0 + r, gk = k0 + c;
      xs[c][r] = (srow[r] >= 0 && gk < K) ? to_f(x[(size_t)srow[r] * ldx + gk]) : 0.0f;
      ws[c][r] = (gn < N && gk < K) ? to_f(w[(size_t)gn * K + gk]) : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < LT_BK; ++c) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { a[i] = xs[c][ty * 4 + i]; b[i] = ws[c][tx * 4 + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx * 4 + j;
      if (gn < N) out[(size_t)gm * ldo + gn] = from_f<OutT>(apply_act(acc[i][j], act, p0, p1));
    }
  }
}

template <typename T, typename OutT>
static int launch_linear(const void* x, int ldx, const void* w, void* out, int ldo, int M, int N, int K, int act, float p0,
                         float p1, cudaStream_t st, bool tensor_cores, LinearGroup g = LinearGroup{0, 0, 0, 1, nullptr, nullptr, nullptr},
                         int nbatch = 1, bool early = false) {
  if (M <= LR_MAXM && g.tile_group == nullptr) {
    constexpr int VN = Vec<T>::N;
    const int vec_ok = (K % VN == 0) && (ldx % VN == 0) && ((uintptr_t)x % 16 == 0) && ((uintptr_t)w % 16 == 0) &&
                       (g.x_bs % VN == 0) && (g.w_bs % VN == 0);
    if constexpr (sizeof(T) == 2) {
      if (tensor_cores && vec_ok && M > 2 && K >= LM_MIN_K && K <= 16 * LM_MAX_SEG && (long)((N + 15) / 16) * nbatch >= (M > 4 ? 96 : 192) &&
          !(M <= 4 && lm_short_tail(N, K, nbatch))) {
        lm_launch<OutT>((const T*)x, ldx, (const T*)w, (OutT*)out, ldo, M, N, K, act, p0, p1, st, g, nbatch);
        return cudaGetLastError() == cudaSuccess ? JL_OK : JL_ERR_CUDA;
      }
      if (vec_ok && nbatch == 1 && g.w_index == nullptr && flow_takes(M, N, K, early))
        return flow_launch<OutT>((const T*)x, ldx, (const T*)w, (OutT*)out, ldo, M, N, K, act, p0, p1, early, st);
    }
    const dim3 blocks((N + LR_ROWS - 1) / LR_ROWS, nbatch);
#define JL_LR(MM)                                                                                                       \
  case MM:                                                                                                              \
    JL_LAUNCH_PDL((linear_rows_kernel<T, OutT, MM>), dim3(blocks), dim3(LR_WARPS * 32), 0, st, (const T*)x, ldx, (const T*)w, (OutT*)out, ldo, N, K, act, \
                                                                   p0, p1, vec_ok, g);                                  \
    break;
    switch (M) { JL_LR(1) JL_LR(2) JL_LR(3) JL_LR(4) JL_LR(5) JL_LR(6) JL_LR(7) JL_LR(8) }
#undef JL_LR
  } else {
    if constexpr (sizeof(T) == 4 && sizeof(OutT) == 4) {
      if (tensor_cores && linear_f32_takes(M, K, ldx, g, x, w))
        return linear_f32_launch((const float*)x, ldx, (const float*)w, (float*)out, ldo, M, N, K, act, p0, p1, st, g, nbatch) == cudaSuccess
                   ? JL_OK : JL_ERR_CUDA;
    }
    dim3 grid((N + LT_BN - 1) / LT_BN, (M + LT_BM - 1) / LT_BM, g.tile_group ? 1 : nbatch);
    JL_LAUNCH_PDL((linear_tiled_kernel<T, OutT>), dim3(grid), dim3(256), 0, st, (const T*)x, ldx, (const T*)w, (OutT*)out, ldo, M, N, K, act, p0, p1, g);
  }
  return cudaGetLastError() == cudaSuccess ? JL_OK : JL_ERR_CUDA;
}

}  // namespace jl

using namespace jl;

static int linear_any(const void* x, int ldx, const void* w, void* out, int ldo, int M, int N, int K, int act, float p0, float p1, int dtype,
                      int out_f32, void* stream, bool tensor_cores, bool early = false) {
  JL_CHECK_ARG(M >= 1 && N >= 1 && K >= 1 && ldx >= K && ldo >= N, "jl_linear_any: bad shape M=%d N=%d K=%d ldx=%d ldo=%d", M, N,
               K, ldx, ldo);
  JL_CHECK_ARG(act >= 0 && act <= ACT_LAST, "jl_linear_any: bad activation %d", act);
  cudaStream_t st = (cudaStream_t)stream;
  const LinearGroup plain{0, 0, 0, 1, nullptr, nullptr, nullptr};
  if (early) {
    // inside one captured graph everything before the graph is complete, whatever wrote the weights included; outside, the kernel just
    // ahead in the stream may have written them
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    early = cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusActive;
  }
  int rc;
  if (dtype == DT_BF16)
    rc = out_f32 ? launch_linear<__nv_bfloat16, float>(x, ldx, w, out, ldo, M, N, K, act, p0, p1, st, tensor_cores, plain, 1, early)
                 : launch_linear<__nv_bfloat16, __nv_bfloat16>(x, ldx, w, out, ldo, M, N, K, act, p0, p1, st, tensor_cores, plain, 1, early);
  else
    rc = launch_linear<float, float>(x, ldx, w, out, ldo, M, N, K, act, p0, p1, st, tensor_cores);
  if (rc != JL_OK) return cuda_fail(cudaGetLastError(), "jl_linear_any launch");
  return JL_OK;
}

extern "C" JL_API int jl_linear_any(const void* x, int ldx, const void* w, void* out, int ldo, int M, int N, int K, int act,
                                    float p0, float p1, int dtype, int out_f32, void* stream) {
  return linear_any(x, ldx, w, out, ldo, M, N, K, act, p0, p1, dtype, out_f32, stream, hybrid_tensor_cores());
}

extern "C" JL_API int jl_linear_resident(const void* x, int ldx, const void* w, void* out, int ldo, int M, int N, int K, int act,
                                         float p0, float p1, int dtype, int out_f32, void* stream) {
  return linear_any(x, ldx, w, out, ldo, M, N, K, act, p0, p1, dtype, out_f32, stream, hybrid_tensor_cores(), true);
}

extern "C" JL_API int jl_linear_exact(const void* x, int ldx, const void* w, void* out, int ldo, int M, int N, int K, int act,
                                      float p0, float p1, int dtype, int out_f32, void* stream) {
  return linear_any(x, ldx, w, out, ldo, M, N, K, act, p0, p1, dtype, out_f32, stream, false);
}

extern "C" JL_API int jl_linear_tile_rows(void) { return LT_BM; }

extern "C" JL_API int jl_linear_grouped(const void* x, int ldx, long long x_bs, const void* w, long long w_bs, void* out, int ldo,
                                        long long o_bs, int nbatch, int x_div, int M, int N, int K, int act, float p0,
                                        float p1, const int* w_index, const int* tile_group, const int* row_src, int dtype, int out_f32,
                                        void* stream) {
  JL_CHECK_ARG(M >= 1 && N >= 1 && K >= 1 && ldx >= K && ldo >= N && nbatch >= 1 && x_div >= 1, "jl_linear_grouped: bad shape M=%d N=%d K=%d ldx=%d ldo=%d",
               M, N, K, ldx, ldo);
  JL_CHECK_ARG(act >= 0 && act <= ACT_LAST, "jl_linear_grouped: bad activation %d", act);
  JL_CHECK_ARG(tile_group == nullptr || M % LT_BM == 0, "jl_linear_grouped: sorted rows come in tiles of %d, M=%d", LT_BM, M);
  JL_CHECK_ARG(nbatch <= 65535, "jl_linear_grouped: %d batches above the grid limit", nbatch);
  cudaStream_t st = (cudaStream_t)stream;
  const LinearGroup g{x_bs, w_bs, o_bs, x_div, w_index, tile_group, row_src};
  const bool tc = hybrid_tensor_cores();
  int rc;
  if (dtype == DT_BF16)
    rc = out_f32 ? launch_linear<__nv_bfloat16, float>(x, ldx, w, out, ldo, M, N, K, act, p0, p1, st, tc, g, nbatch)
                 : launch_linear<__nv_bfloat16, __nv_bfloat16>(x, ldx, w, out, ldo, M, N, K, act, p0, p1, st, tc, g, nbatch);
  else
    rc = launch_linear<float, float>(x, ldx, w, out, ldo, M, N, K, act, p0, p1, st, tc, g, nbatch);
  if (rc != JL_OK) return cuda_fail(cudaGetLastError(), "jl_linear_grouped launch");
  return JL_OK;
}

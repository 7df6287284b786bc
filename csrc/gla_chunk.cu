// Prompts of gated linear attention S_t = diag(alpha_t) S_(t-1) + k_t v_tᵀ, o_t = S_tᵀ q_t with projected decays, 64 tokens at a time on the tensor cores, with fp32 accuracy.
//
// Within a chunk that starts from the state S, with A_i = alpha_1 ... alpha_i per key channel,
//     o_i = (A_i q_i)·S + sum_{j<=i} P_ij v_j,     P_ij = sum_d q_i[d] k_j[d] alpha_(j+1)[d] ... alpha_i[d],
//     S  <- A_64 S + sum_j (alpha_(j+1) ... alpha_64 k_j) v_jᵀ.
// Products of decays are running products, never quotients.  P is formed by halves: pairs inside a block of 8 tokens one decay at a time; a block of 2 L
// tokens is two blocks of L whose cross terms are (decays from the right block's start · q_i) · (k_j · decays to the left block's end), and the two
// factors grow with L in place until they are A q over the chunk.
//   gla_chunk_state_kernel  (chunk, head, row): decays (kept for the second kernel), sum_j (..k_j) v_jᵀ and A_64;
//   gla_combine_kernel      walks the chunks: the state every chunk starts from;
//   gla_chunk_out_kernel    (chunk, head, row): P, then the two products of o.
// The products of 64 k are tcgen05 MMAs of bfloat16 parts, three per fp32 number and six products (linear_f32.cuh; a chunk's state sum in four sums of 16 tokens, as it is
// what the following chunks inherit and the tensor core cuts off where it adds), value columns as the MMA's 128 rows
// (tokens or key channels lie along K as they come: MN-major operands); P's cross terms are the same on mma.sync.  What comes out infinite or NaN is
// formed again token by token, so that nothing of a token that is not finite reaches an earlier one.
// Bound: latencies of a CTA's chain of phases (loads, decays, pairs and factors, cross terms, two rounds of tensor core, stores) with two CTAs per SM: 21 % of the warps are active, half
// of the issue slots, 5 and 13 % of the tensor pipe are used, 105 and 130 MB pass the L2 (2048 tokens x 16 heads of 64 x 128).  One B200, us, walking twice over chunks of tokens
// (gla_scan.cu) -> this, all launches of the scan: 2048 tokens x 16 heads of 64 x 128 123 -> 77 (a layer of width 2048 199 -> 149), 2 rows x 1000 120 -> 73, 500 89 -> 30, 4 rows x
// 512 x 8 heads of 32 x 64 68 -> 34, 4 rows x 128 x 16 heads of 128 x 128 101 -> 53.
// Error against float64 (2-norm of the read-outs; of the state), the decays' own included, walk -> this: decays of 0.99 in the mean, 65 tokens 2.2e-7; 2.7e-7 -> 1.9e-7; 2.6e-7, 500
// 1.01e-6; 1.53e-6 -> 9.5e-7; 1.49e-6, 2048 2.30e-6; 3.14e-6 -> 2.25e-6; 3.17e-6; operands of one sign, 65 8.8e-8; 2.4e-7 -> 5.7e-8; 2.2e-7, 500 6.5e-7; 1.82e-6 -> 5.4e-7; 1.78e-6, 2048
// 1.70e-6; 5.93e-6 -> 1.59e-6; 5.99e-6.  Decays of 0.72, where few tokens are summed and the cut-off shows: 500 1.04e-7; 8.3e-8 -> 1.07e-7; 8.9e-8, of one sign 5.4e-8; 9.0e-8 ->
// 5.9e-8; 8.7e-8.
#include "gla_scan.cuh"
#include "jllama_b200.h"
#include "linear_f32.cuh"
#include "seq_types.cuh"
#include "tcgen05.cuh"

namespace jl {

constexpr int GC_T = 64, GC_THREADS = 256, GC_DV = 128;                  // tokens of a chunk; value columns of a CTA
constexpr uint32_t GC_TILE = GC_T * 128;                                  // 64 rows of 64 bf16
constexpr uint32_t GC_V_BYTES = 3 * 2 * GC_TILE, GC_K_BYTES = 3 * GC_TILE;
constexpr int GC_PP = GC_T + 8, GC_R = 32;                               // (GC_R: of the decays' low-rank input at a time)
// parts of the six products, the smallest first
__host__ __device__ constexpr int gc_a(int q) { return 0x010120 >> (4 * q) & 15; }
__host__ __device__ constexpr int gc_b(int q) { return 0x001102 >> (4 * q) & 15; }

struct GlaChunk {
  GlaParams p;
  float* alpha;                        // [B*S][H][D]
};

__device__ __forceinline__ int gc_first(const GlaParams& p, int b) { return max(0, (p.pad_left ? p.pad_left[b] : 0) - (p.cache_len ? *p.cache_len : 0)); }

__device__ __forceinline__ float2 gc_qk(const GlaParams& p, size_t m, int h, int d) {
  const float* row = p.y + m * p.ldy + h * p.D + d;
  return make_float2(row[p.q_off] * p.q_scale, row[p.k_off] * p.k_scale);
}
__device__ __forceinline__ float gc_value(const GlaParams& p, size_t m, int h, int c) { return c < p.Dv ? p.y[m * p.ldy + p.v_off + h * p.Dv + c] : 0.0f; }

__device__ __forceinline__ void gc_store16(uint32_t at, const uint4& v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// eight columns of a row of a [64][128] tile -> three bfloat16 parts of two 64-column tiles (128-byte rows, swizzled)
__device__ __forceinline__ void gc_put8(uint32_t dst, int row, int c, const float4& a, const float4& b) {
  uint4 part[3];
  lf_split8(a, b, part);
  const uint32_t at = dst + (c >> 3) * GC_TILE + row * 128 + (((c & 7) ^ (row & 7)) << 4);
#pragma unroll
  for (int q = 0; q < 3; ++q) gc_store16(at + q * 2 * GC_TILE, part[q]);
}
// A [64][128] tile whose row r lies at src + min(r, rows - 1) * pitch; rows outside [lo, hi) and columns from `cols` on are zero.  `wide`: whole pieces of
// eight, all asked for by load() and used by put(); else value(row, column) one by one in put().
struct GcTile {
  float4 a[4], b[4];
  __device__ __forceinline__ void load(bool wide, const float* src, int pitch, int rows, int cols) {
    if (!wide) return;
    const float* from = src + min((int)threadIdx.x % 16 * 8, max(cols - 8, 0));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float* r = from + min((int)threadIdx.x / 16 + 16 * i, rows - 1) * pitch;
      a[i] = *reinterpret_cast<const float4*>(r);
      b[i] = *reinterpret_cast<const float4*>(r + 4);
    }
  }
  template <typename F>
  __device__ __forceinline__ void put(uint32_t dst, bool wide, int cols, int lo, int hi, F&& value) {
    const int c = threadIdx.x % 16, r0 = threadIdx.x / 16;
    if (wide) {
      const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = r0 + 16 * i;
        const bool in = row >= lo && row < hi && c * 8 < cols;
        gc_put8(dst, row, c, in ? a[i] : zero, in ? b[i] : zero);
      }
      return;
    }
#pragma unroll 1
    for (int row = r0; row < GC_T; row += 16) {
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = row >= lo && row < hi && c * 8 + e < cols ? value(row, c * 8 + e) : 0.0f;
      gc_put8(dst, row, c, make_float4(v[0], v[1], v[2], v[3]), make_float4(v[4], v[5], v[6], v[7]));
    }
  }
};

template <typename T, int DB>
__global__ void __launch_bounds__(GC_THREADS, DB == 1 ? 2 : 1) gla_chunk_state_kernel(const __grid_constant__ GlaChunk g, const T* __restrict__ a2,
                                                                        const T* __restrict__ a2b, int wide) {
  const GlaParams& p = g.p;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(8) unsigned long long bar_mem;
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(16) float prod[4][64];
  const uint32_t raw = tc::smem_u32(smem_raw), base = (raw + 1023u) & ~1023u, bar = tc::smem_u32(&bar_mem);
  const uint32_t sv = base, sk = base + GC_V_BYTES;
  float* ks = reinterpret_cast<float*>(smem_raw + (base - raw) + GC_V_BYTES + DB * GC_K_BYTES);           // [64][64] keys | decays (first their logits)
  float* as = ks + GC_T * 64;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nv = (p.Dv + GC_DV - 1) / GC_DV, h = blockIdx.y / nv, c0 = blockIdx.y % nv * GC_DV, b = blockIdx.z, chunk = blockIdx.x;
  if (warp == 0) {
    tc::tmem_alloc(tc::smem_u32(&tmem_slot), 256 * DB);
    if (lane == 0) { tc::mbar_init(bar, 1); tc::fence_barrier_init(); }
  }
  pdl_wait();
  const int t0 = chunk * GC_T, first = gc_first(p, b);
  const int rows = min(GC_T, p.S - t0);                                     // tokens of the chunk that exist
  const int lo = max(0, first - t0), hi = rows;                             // ... that are real
  const size_t m0 = (size_t)b * p.S + t0;
  GcTile values;
  values.load(wide != 0, p.y + m0 * p.ldy + p.v_off + h * p.Dv + c0, p.ldy, rows, p.Dv - c0);
  const int quarter = tid >> 6, dl = tid & 63;                              // a thread has one channel of 16 tokens
#pragma unroll 1
  for (int db = 0; db < DB; ++db) {
    const int d = db * 64 + dl, dc = min(d, p.D - 1);
    float* kt = ks + quarter * 16 * 64 + dl;
    float* at = as + quarter * 16 * 64 + dl;
    // logits of projected decays: bias + A2 z, GC_R columns of z and rows of A2 at a time in the place of this block's parts of the keys; a round's loads are
    // under way before anything is waited for (one by one they took half of this kernel)
    float* zs = reinterpret_cast<float*>(smem_raw + (base - raw) + GC_V_BYTES + db * GC_K_BYTES);          // [64][GC_R + 1] z, then A2
    float* ws = zs + GC_T * (GC_R + 1);
    float zr[8], wr[8];
    auto ask = [&](int r0) {
      const int r = r0 + lane;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int t = warp + 8 * i;
        zr[i] = r < p.R ? p.y[(m0 + min(t, rows - 1)) * p.ldy + p.a_off + r] : 0.0f;
        wr[i] = r < p.R ? to_f(a2[(size_t)(h * p.D + min(db * 64 + t, p.D - 1)) * p.R + r]) : 0.0f;
      }
    };
    ask(0);
    float v[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      const int s = min(quarter * 16 + t, rows - 1);
      v[t] = gc_qk(p, m0 + s, h, dc).y;
    }
    {
      float a[16];
      const float bias = to_f(a2b[h * p.D + dc]);
#pragma unroll
      for (int t = 0; t < 16; ++t) a[t] = bias;
#pragma unroll 1
      for (int r0 = 0; r0 < p.R; r0 += GC_R) {
        if (r0 > 0) { __syncthreads(); ask(r0); }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          zs[(warp + 8 * i) * (GC_R + 1) + lane] = zr[i];
          ws[(warp + 8 * i) * (GC_R + 1) + lane] = wr[i];
        }
        __syncthreads();
        const int nr = min(GC_R, p.R - r0);
#pragma unroll 4
        for (int r = 0; r < nr; ++r) {
          const float w = ws[dl * (GC_R + 1) + r];
#pragma unroll
          for (int t = 0; t < 16; ++t) a[t] = fmaf(w, zs[(quarter * 16 + t) * (GC_R + 1) + r], a[t]);
        }
      }
#pragma unroll
      for (int t = 0; t < 16; ++t) at[t * 64] = a[t];
    }
#pragma unroll
    for (int t = 0; t < 16; ++t) kt[t * 64] = v[t];
    if (db == 0) {
      values.put(sv, wide != 0, p.Dv - c0, lo, hi, [&](int row, int c) { return gc_value(p, m0 + row, h, c0 + c); });
      __syncthreads();
      pdl_launch_dependents();                                              // (this CTA has its tensor memory)
    }
    // keys times the decays behind them, in the quarter and then in the chunk
    float all = 1.0f;
#pragma unroll 4
    for (int t = 15; t >= 0; --t) {
      const int s = quarter * 16 + t;
      const bool in = s >= lo && s < hi && d < p.D;
      const float a = expf(log_sigmoid(at[t * 64]) * p.inv_tau);
      if (in && c0 == 0) g.alpha[((m0 + s) * p.H + h) * p.D + d] = a;
      kt[t * 64] = in ? kt[t * 64] * all : 0.0f;
      if (in) all *= a;
    }
    prod[quarter][dl] = all;
    __syncthreads();
    if (quarter == 0 && c0 == 0 && d < p.D)
      p.cdecay[(((size_t)b * p.NC + chunk) * p.H + h) * p.D + d] = all * (prod[1][dl] * (prod[2][dl] * prod[3][dl]));
#pragma unroll
    for (int i = 0; i < 2; ++i) {                                           // the parts, eight channels of a token a piece
      const int s = tid / 8 + 32 * i, c = tid % 8;
      float4 x = *reinterpret_cast<const float4*>(ks + s * 64 + c * 8), y = *reinterpret_cast<const float4*>(ks + s * 64 + c * 8 + 4);
#pragma unroll
      for (int q = 1; q < 4; ++q)
        if (q > s / 16) {
          const float4 u = *reinterpret_cast<const float4*>(&prod[q][c * 8]), w = *reinterpret_cast<const float4*>(&prod[q][c * 8 + 4]);
          x = make_float4(x.x * u.x, x.y * u.y, x.z * u.z, x.w * u.w);
          y = make_float4(y.x * w.x, y.y * w.y, y.z * w.z, y.w * w.w);
        }
      uint4 part[3];
      lf_split8(x, y, part);
#pragma unroll
      for (int q = 0; q < 3; ++q) gc_store16(sk + db * GC_K_BYTES + q * GC_TILE + s * 128 + ((c ^ (s & 7)) << 4), part[q]);
    }
    if (db + 1 < DB) __syncthreads();                                       // (prod and the channels of the next block)
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  if (warp == 0) {
    if (tc::elect_one()) {
      constexpr uint32_t IDESC = tc::idesc_bf16_f32(GC_DV, 64, true, true);
      const uint64_t dv = tc::smem_desc_mnmajor_sw128(sv, GC_TILE, 1024), dk = tc::smem_desc_mnmajor_sw128(sk, GC_TILE, 1024);
#pragma unroll
      for (int db = 0; db < DB; ++db)
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int q = 0; q < 6; ++q)
            tc::mma_ss(tmem + (k * DB + db) * 64, dv + ((gc_a(q) * 2 * GC_TILE + k * 2048) >> 4), dk + ((db * GC_K_BYTES + gc_b(q) * GC_TILE + k * 2048) >> 4), IDESC,
                       q != 0);
      tc::mma_commit(bar);
    }
    __syncwarp();
  }
  tc::mbar_wait(bar, 0);
  tc::fence_after_sync();
  // lanes are value columns: two groups of four warps take the halves of the key channels
  const int c = c0 + (warp & 3) * 32 + lane;
  float* out = p.cstate + (((size_t)b * p.NC + chunk) * p.H + h) * p.D * p.Dv + c;
#pragma unroll 1
  for (int e0 = (warp >> 2) * 32 * DB; e0 < ((warp >> 2) + 1) * 32 * DB; e0 += 32) {
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; i += 16) {
      uint32_t u[4][16];
#pragma unroll
      for (int k = 0; k < 4; ++k) tc::tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + k * 64 * DB + e0 + i, u[k]);
      tc::tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j)
        v[i + j] = (__uint_as_float(u[0][j]) + __uint_as_float(u[1][j])) + (__uint_as_float(u[2][j]) + __uint_as_float(u[3][j]));
    }
    if (c < p.Dv) {
      bool bad = false;
#pragma unroll
      for (int e = 0; e < 32; ++e)
        if (e0 + e < p.D) {
          out[(size_t)(e0 + e) * p.Dv] = v[e];
          bad |= !(fabsf(v[e]) < INFINITY);
        }
      if (bad)
#pragma unroll 1
        for (int d = e0; d < min(e0 + 32, p.D); ++d) {
          if (fabsf(out[(size_t)d * p.Dv]) < INFINITY) continue;
          float s = 0.0f;
#pragma unroll 1
          for (int t = lo; t < hi; ++t) {
            float a;
            if (c0 > 0) {                                       // (the first slice's CTAs may not have stored them yet)
              const int n = h * p.D + d;
              a = to_f(a2b[n]);
              for (int r = 0; r < p.R; ++r) a = fmaf(to_f(a2[(size_t)n * p.R + r]), p.y[(m0 + t) * p.ldy + p.a_off + r], a);
              a = expf(log_sigmoid(a) * p.inv_tau);
            } else {
              a = g.alpha[((m0 + t) * p.H + h) * p.D + d];
            }
            s = fmaf(a, s, gc_qk(p, m0 + t, h, d).y * gc_value(p, m0 + t, h, c));
          }
          out[(size_t)d * p.Dv] = s;
        }
    }
    __syncwarp();
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 256 * DB);
}

__device__ __forceinline__ void gc_mma16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void gc_split2(const float2 v, uint32_t (&part)[3]) {
  part[0] = pack_bf16(v.x, v.y);
  const float x = v.x - bf16_lo(part[0]), y = v.y - bf16_hi(part[0]);
  part[1] = pack_bf16(x, y);
  part[2] = pack_bf16(x - bf16_lo(part[1]), y - bf16_hi(part[1]));
}

// Shared memory of the second kernel, in bytes: the cross terms' factors of the three levels, 32 rows of q and of k each (then the state, then the values, in
// three parts) | P | sums inside blocks of 8 | products of the decays | A q (then P) in three parts.  Two CTAs per SM: what a chunk takes is latency.
constexpr int GC_PITCH = 72;                                                // floats of a row of 64: rows of a fragment load on distinct banks
struct GcOut {
  static constexpr uint32_t LEVEL = 32 * GC_PITCH * 4;
  static constexpr uint32_t W = 0, P = 6 * LEVEL, DIAG = P + GC_T * GC_PP * 4, PROD = DIAG + 2 * 8 * 36 * 4;
  static constexpr uint32_t XQ = (PROD + 4 * 64 * 4 + 1023) / 1024 * 1024, BYTES = XQ + GC_K_BYTES + 1024;
  static_assert(6 * LEVEL >= GC_V_BYTES, "state and values in the factors' place");
};

__global__ void __launch_bounds__(GC_THREADS, 2) gla_chunk_out_kernel(const __grid_constant__ GlaChunk g, int wide) {
  const GlaParams& p = g.p;
  using L = GcOut;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(8) unsigned long long bar_mem;
  __shared__ uint32_t tmem_slot;
  const uint32_t raw = tc::smem_u32(smem_raw), base = (raw + 1023u) & ~1023u, bar = tc::smem_u32(&bar_mem);
  uint8_t* mem = smem_raw + (base - raw);
  float* wq = reinterpret_cast<float*>(mem + L::W);                         // [level][32][GC_PITCH], then the keys'
  float* wk = wq + 3 * 32 * GC_PITCH;
  float* pf = reinterpret_cast<float*>(mem + L::P);                         // [i][j], pitch GC_PP
  float* diag = reinterpret_cast<float*>(mem + L::DIAG);                    // [half of the channels][block of 8][pair]
  float* prod = reinterpret_cast<float*>(mem + L::PROD);                    // [4][64]: decays of 16 tokens
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nv = (p.Dv + GC_DV - 1) / GC_DV, h = blockIdx.y / nv, c0 = blockIdx.y % nv * GC_DV, b = blockIdx.z, chunk = blockIdx.x;
  const int blocks = (p.D + 63) / 64;                                       // of 64 channels: one or two
  const uint32_t cols = blocks == 1 ? 128u : 256u;
  if (warp == 0) {
    tc::tmem_alloc(tc::smem_u32(&tmem_slot), cols);
    if (lane == 0) { tc::mbar_init(bar, 1); tc::fence_barrier_init(); }
  }
  for (int i = tid; i < GC_T * GC_PP; i += GC_THREADS) pf[i] = 0.0f;
  pdl_wait();
  const int t0 = chunk * GC_T, first = gc_first(p, b);
  const int rows = min(GC_T, p.S - t0);                                     // tokens of the chunk that exist
  const int lo = max(0, first - t0), hi = rows;                             // ... that are real
  const size_t m0 = (size_t)b * p.S + t0;
  const float* s_in = p.cstate + (((size_t)b * p.NC + chunk) * p.H + h) * p.D * p.Dv;
  const bool s_wide = p.Dv % 8 == 0 && ((uintptr_t)p.cstate & 15) == 0;
  const int quarter = tid >> 6, dl = tid & 63;                              // a thread has one channel of 16 tokens
  constexpr uint32_t IDESC = tc::idesc_bf16_f32(GC_DV, 64, true, false);
  int phase = 0;
  auto visible = [&] {                                                      // writes so far -> tensor core
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
  };
  auto product = [&](uint32_t left, uint32_t right, uint32_t d) {           // 64 k: columns x tokens
    if (warp == 0) {
      if (tc::elect_one()) {
        const uint64_t da = tc::smem_desc_mnmajor_sw128(left, GC_TILE, 1024), db = tc::smem_desc_kmajor_sw128(right);
#pragma unroll
        for (int q = 0; q < 6; ++q)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            tc::mma_ss(d, da + ((gc_a(q) * 2 * GC_TILE + k * 2048) >> 4), db + ((gc_b(q) * GC_TILE + k * 32) >> 4), IDESC, q != 0 || k != 0);
        tc::mma_commit(bar);
      }
      __syncwarp();
    }
  };
  auto finished = [&] { tc::mbar_wait(bar, phase); tc::fence_after_sync(); phase ^= 1; };
  GcTile tile;
#pragma unroll 1
  for (int db = 0; db < blocks; ++db) {
    const int d = db * 64 + dl, dc = min(d, p.D - 1);
    const float* decay = g.alpha + (m0 * p.H + h) * p.D + dc;
    float q[16], k[16], a[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      const int s = min(quarter * 16 + t, rows - 1);
      const float2 v = gc_qk(p, m0 + s, h, dc);
      q[t] = v.x; k[t] = v.y;
      a[t] = decay[(size_t)s * p.H * p.D];
    }
    float p0 = 1.0f, p1 = 1.0f;                                             // decays of the first and the last eight tokens
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      const int s = quarter * 16 + t;
      const bool in = s >= lo && s < hi && d < p.D;
      q[t] = in ? q[t] : 0.0f; k[t] = in ? k[t] : 0.0f; a[t] = in ? a[t] : 1.0f;
      if (t < 8) p0 *= a[t]; else p1 *= a[t];
    }
    if (db > 0) finished();                                                 // (its operands are done with)
    prod[quarter * 64 + dl] = p0 * p1;
    __syncthreads();
    if (db == 0) pdl_launch_dependents();                                   // (this CTA has its tensor memory)
    // pairs inside blocks of 8, one decay at a time; the 32 channels of a warp meet by shuffles: at each step a lane keeps half of its sums and gives the
    // other half to its partner, so that lane n ends with pair n, and four lanes with the last four
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float v[36];
#pragma unroll
      for (int j = 0, n = 0; j < 8; ++j) {
        float r = k[e * 8 + j];
#pragma unroll
        for (int i = j; i < 8; ++i, ++n) {
          if (i > j) r *= a[e * 8 + i];
          v[n] = q[e * 8 + i] * r;
        }
      }
      float* to = diag + ((warp & 1) * 8 + quarter * 2 + e) * 36;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < o; ++i) {
          const float keep = up ? v[i + o] : v[i], give = up ? v[i] : v[i + o];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
      }
      to[lane] = v[0];
#pragma unroll
      for (int o = 16, n = 2; n > 0; o >>= 1, n >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
          const float keep = up ? v[32 + i + n] : v[32 + i], give = up ? v[32 + i] : v[32 + i + n];
          v[32 + i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) v[32] += __shfl_xor_sync(0xffffffffu, v[32], o);
      if ((lane & 7) == 0) to[32 + (lane >> 4) * 2 + ((lane >> 3) & 1)] = v[32];
    }
    // the factors: queries times the decays since their block's start, keys times those to its end, blocks of 8, 16, 32 and (queries) 64 tokens
#pragma unroll
    for (int e = 0; e < 16; e += 8) {
      float pre = 1.0f, suf = 1.0f;
#pragma unroll
      for (int t = 0; t < 8; ++t) { pre *= a[e + t]; q[e + t] *= pre; }
#pragma unroll
      for (int t = 7; t >= 0; --t) { k[e + t] *= suf; suf *= a[e + t]; }
    }
    const float left = prod[(quarter ^ 1) * 64 + dl];                       // the other quarter of this half
    const float half0 = prod[dl] * prod[64 + dl];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      wq[(quarter * 8 + t) * GC_PITCH + dl] = q[8 + t];
      wk[(quarter * 8 + t) * GC_PITCH + dl] = k[t];
      q[8 + t] *= p0;
      k[t] *= p1;
    }
    {
      const bool odd = (quarter & 1) != 0, upper = quarter >= 2;
      float* w1 = (odd ? wq : wk) + (32 + (quarter >> 1) * 16) * GC_PITCH + dl;
      float* w2 = (upper ? wq : wk) + (64 + (quarter & 1) * 16) * GC_PITCH + dl;
      const float ql = odd ? left : 1.0f, kl = odd ? 1.0f : left, qh = upper ? half0 : 1.0f;
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        w1[t * GC_PITCH] = odd ? q[t] : k[t];
        q[t] *= ql;
        k[t] *= kl;
        w2[t * GC_PITCH] = upper ? q[t] : k[t];
        const int s = quarter * 16 + t;
        const uint32_t to = base + L::XQ + s * 128 + (((dl >> 3) ^ (s & 7)) << 4) + (dl & 7) * 2;
        float x = q[t] * qh;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          const __nv_bfloat16 part = __float2bfloat16(x);
          asm volatile("st.shared.u16 [%0], %1;" ::"r"(to + e * GC_TILE), "h"(__bfloat16_as_ushort(part)) : "memory");
          x -= __bfloat162float(part);
        }
      }
    }
    __syncthreads();
    const float* src = s_in + (size_t)db * 64 * p.Dv + c0;                  // 64 key channels of the state the chunk starts from
    const int n = min(GC_T, p.D - db * 64);
    tile.load(s_wide, src, p.Dv, n, p.Dv - c0);
    for (int x = tid; x < 8 * 36; x += GC_THREADS) {
      const int blk = x / 36, e = x % 36;
      const int j = (e >= 8) + (e >= 15) + (e >= 21) + (e >= 26) + (e >= 30) + (e >= 33) + (e >= 35), i = e - (8 * j - j * (j - 1) / 2) + j;
      pf[(blk * 8 + i) * GC_PP + blk * 8 + j] += diag[blk * 36 + e] + diag[(8 + blk) * 36 + e];
    }
    // cross terms, two 16 x 8 tiles a warp: one of the two blocks of 32, and one of the four pairs of 8 or the two of 16
#pragma unroll 1
    for (int i = 0; i < 2; ++i) {
      const int gr = lane >> 2, cc = (lane & 3) * 2;
      const int lev = i == 0 ? 2 : warp < 4 ? 0 : 1, w4 = warp & 3;
      const int qr = lev == 2 ? 64 + (warp >> 2) * 16 : lev == 1 ? 32 + (w4 >> 1) * 16 : w4 * 8;
      const int kr = lev == 2 ? 64 + w4 * 8 : lev == 1 ? 32 + w4 * 8 : w4 * 8;
      const int r0 = lev == 2 ? 32 + (warp >> 2) * 16 : lev == 1 ? (w4 >> 1) * 32 + 16 : w4 * 16 + 8;
      const int j0 = lev == 2 ? w4 * 8 : lev == 1 ? (w4 >> 1) * 32 + (w4 & 1) * 8 : w4 * 16;
      float sum[2][4] = {};                                                 // of 32 channels each
#pragma unroll
      for (int kh = 0; kh < 2; ++kh) {
        uint32_t fa[2][3][4], fb[2][3][2];
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
          const int at = (kh * 2 + kk) * 16 + cc;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            // (the pairs of 8 have eight rows: the other half of the tile repeats them and is not stored)
            uint32_t part[3];
            gc_split2(*reinterpret_cast<const float2*>(wq + (qr + gr + (lev > 0 ? (e & 1) * 8 : 0)) * GC_PITCH + at + (e >> 1) * 8), part);
#pragma unroll
            for (int x = 0; x < 3; ++x) fa[kk][x][e] = part[x];
          }
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            uint32_t part[3];
            gc_split2(*reinterpret_cast<const float2*>(wk + (kr + gr) * GC_PITCH + at + e * 8), part);
#pragma unroll
            for (int x = 0; x < 3; ++x) fb[kk][x][e] = part[x];
          }
        }
#pragma unroll
        for (int x = 0; x < 6; ++x)
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) gc_mma16816(sum[kh], fa[kk][gc_a(x)], fb[kk][gc_b(x)]);
      }
      float* to = pf + (r0 + gr) * GC_PP + j0 + cc;
      to[0] += sum[0][0] + sum[1][0]; to[1] += sum[0][1] + sum[1][1];
      if (lev > 0) { to[8 * GC_PP] += sum[0][2] + sum[1][2]; to[8 * GC_PP + 1] += sum[0][3] + sum[1][3]; }
    }
    __syncthreads();
    tile.put(base + L::W, s_wide, p.Dv - c0, 0, n, [&](int row, int c) { return src[(size_t)row * p.Dv + c]; });
    visible();
    product(base + L::W, base + L::XQ, tmem_slot + db * 64);
  }
  tile.load(wide != 0, p.y + m0 * p.ldy + p.v_off + h * p.Dv + c0, p.ldy, rows, p.Dv - c0);      // the values
  finished();                                                               // (and every thread has seen this phase of the barrier before the next can end)
  tile.put(base + L::W, wide != 0, p.Dv - c0, lo, hi, [&](int row, int c) { return gc_value(p, m0 + row, h, c0 + c); });
#pragma unroll
  for (int i = 0; i < 2; ++i) {                                             // P [64][64] -> three K-major tiles
    const int row = tid / 8 + 32 * i, c = tid % 8;
    const float4 u = *reinterpret_cast<const float4*>(pf + row * GC_PP + c * 8), v = *reinterpret_cast<const float4*>(pf + row * GC_PP + c * 8 + 4);
    uint4 part[3];
    lf_split8(u, v, part);
#pragma unroll
    for (int q = 0; q < 3; ++q) gc_store16(base + L::XQ + q * GC_TILE + row * 128 + ((c ^ (row & 7)) << 4), part[q]);
  }
  visible();
  const uint32_t tmem = tmem_slot;
  product(base + L::W, base + L::XQ, tmem + blocks * 64);
  finished();
  const int c = c0 + (warp & 3) * 32 + lane, s0 = (warp >> 2) * 32;
  const uint32_t row = tmem + ((uint32_t)((warp & 3) * 32) << 16) + s0;
  float o[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) o[i] = 0.0f;
#pragma unroll 1
  for (int db = 0; db <= blocks; ++db) {
    uint32_t v[32];
    tc::tmem_ld32(row + db * 64, v);
    tc::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; ++i) o[i] += __uint_as_float(v[i]);
  }
  if (c < p.Dv) {
    const size_t step = (size_t)p.H * p.Dv;
    float* out = p.o + (m0 * p.H + h) * p.Dv + c;
    float* to = out + s0 * step;
    bool bad = false;
#pragma unroll
    for (int i = 0; i < 32; ++i, to += step) {
      const bool in = s0 + i >= lo;
      if (s0 + i < hi) *to = in ? o[i] : 0.0f;
      bad |= in && !(fabsf(o[i]) < INFINITY);
    }
    if (bad) {                                                              // the column's state, token by token from the chunk's start
      float st[128];
#pragma unroll 1
      for (int d = 0; d < p.D; ++d) st[d] = s_in[(size_t)d * p.Dv + c];
#pragma unroll 1
      for (int t = lo; t < min(s0 + 32, hi); ++t) {
        const float v = gc_value(p, m0 + t, h, c);
        float acc = 0.0f;
#pragma unroll 1
        for (int d = 0; d < p.D; ++d) {
          const float2 qk = gc_qk(p, m0 + t, h, d);
          st[d] = fmaf(g.alpha[((m0 + t) * p.H + h) * p.D + d], st[d], qk.y * v);
          acc = fmaf(qk.x, st[d], acc);
        }
        if (t >= s0 && !(fabsf(out[t * step]) < INFINITY)) out[t * step] = acc;
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, cols);
}

static int gc_chunks(int S) { return (S + GC_T - 1) / GC_T; }

// Up to 128 key channels, from the tokens on where three launches of parallel chunks beat the walk of gla_scan.cu.  us, walk -> this: D 64 x Dv 128: 1 row x 16 heads 40 tokens 21.8 -> 23.3,
// 48 24.1 -> 21.9, 64 29.9 -> 21.9, 2 rows 48 27.9 -> 23.3, 64 33.7 -> 23.4; 4 rows x 16 heads of 32 x 64, 48 tokens 25.3 -> 21.6; 128 x 128: 1 row x 4 heads 64 tokens 35.4 -> 39.2, 80
// 42.2 -> 34.1, 200 61.3 -> 34.9, 4 rows x 8 heads 40 39.9 -> 41.6, 48 41.3 -> 37.6.
// Decays that are given (one per head, or per token and head) always walk: nothing of their own covers what the tensor core cuts off and the roundings of products of 64 decays.  Error
// against float64 (2-norm of the read-outs), walk -> this: one fixed decay of 0.9, operands of one sign, 500 tokens x 16 heads of 64 x 128 4.1e-8 -> 9.4e-8, decay 1 4.7e-8 ->
// 1.4e-7; a float32 retention layer of 3 x 608 tokens, its state 1.18e-6 -> 1.49e-6; 40 drawn float32 state space layers, their states 9 % further
// off in the mean and 19 % at most (what is cut off has the sign of what the projections before lose), outputs 0 and 4 %.
// Narrow heads, which are padded to 64 (128) channels and 128 columns here and not there: keys of 16 channels from 64 tokens on (4 rows x 4 heads of 16 x 64, 48 tokens 18.1 -> 21.0, 64 22.2 -> 21.0); once the
// chunks fill the SMs several times the walk has them (4 rows x 16 heads, 1000 tokens of 16 x 64 91 -> 100, of 32 x 16 94 -> 98, 400 tokens of 100 x 32 97 -> 112, of 128 x 16 76 -> 111; of
// 128 x 64 and 64 x 64 this).
bool gla_chunk_takes(int B, int S, int H, int D, int Dv) {
  const long slices = (Dv + GC_DV - 1) / GC_DV, ctas = (long)B * H * gc_chunks(S) * slices;
  if (D > 128 || H * slices > 65535 || B > 65535) return false;
  if (D <= 64) return S >= (D <= 16 ? 64 : 48) && !(ctas > 6 * SMS && (D <= 16 || D * Dv < 1024));
  return S >= (B * H < 32 || Dv < 32 ? 80 : Dv < 64 ? 56 : 48) && !(ctas > 2 * SMS && Dv <= 32);
}

size_t gla_chunk_ws_floats(int B, int S, int H, int D, int Dv) {
  const size_t states = (size_t)B * gc_chunks(S) * H * D;
  return states * Dv + (states + 3) / 4 * 4 + (size_t)B * S * H * D;
}

template <int DB>
static int gc_launch(const GlaChunk& g, const void* a2, const void* a2_bias, int dtype, int wide, cudaStream_t st) {
  const GlaParams& p = g.p;
  const dim3 grid(p.NC, p.H * ((p.Dv + GC_DV - 1) / GC_DV), p.B);
  const size_t smem = GC_V_BYTES + DB * GC_K_BYTES + 2 * GC_T * 64 * 4 + 1024;
  JL_DISPATCH_DTYPE(dtype, JL_CUDA(cudaFuncSetAttribute((gla_chunk_state_kernel<T, DB>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
                    JL_CUDA(launch_pdl((gla_chunk_state_kernel<T, DB>), grid, dim3(GC_THREADS), smem, st, g, (const T*)a2, (const T*)a2_bias, wide)));
  JL_CUDA(cudaFuncSetAttribute(gla_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GcOut::BYTES));
  const size_t total = (size_t)p.B * p.H * p.D * p.Dv;
  JL_CUDA(launch_pdl(gla_combine_kernel, dim3((unsigned)((total + 255) / 256 < 1184 ? (total + 255) / 256 : 1184)), dim3(256), 0, st, p));
  JL_CUDA(launch_pdl(gla_chunk_out_kernel, grid, dim3(GC_THREADS), GcOut::BYTES, st, g, wide));
  return JL_OK;
}

int gla_chunk_launch(GlaParams p, const void* a2, const void* a2_bias, float* ws, int dtype, cudaStream_t st) {
  p.NC = gc_chunks(p.S);
  p.L = GC_T;
  const size_t states = (size_t)p.B * p.NC * p.H * p.D;
  p.cstate = ws;
  p.cdecay = ws + states * p.Dv;
  const GlaChunk g{p, p.cdecay + (states + 3) / 4 * 4};
  const int wide = p.Dv % 8 == 0 && p.ldy % 4 == 0 && p.v_off % 4 == 0 && ((uintptr_t)p.y & 15) == 0;
  return p.D <= 64 ? gc_launch<1>(g, a2, a2_bias, dtype, wide, st) : gc_launch<2>(g, a2, a2_bias, dtype, wide, st);
}

}  // namespace jl

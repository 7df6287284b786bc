// One-launch decode attention: RoPE(q, k_new) + KV-cache append + split-KV GQA attention + split merge.
//
// Replaces three launches of the unfused path (rope_kv_kernel → decode_attn_kernel → attn_combine_kernel)
// per layer; at batch 1 those launches cost more than the 8 MB of K/V they move.  Differences from
// decode_attn.cu:
//   * q and the new token's k, v are read straight from the fused qkv activation; the rotation is applied
//     in registers from the fp32 cos/sin table (position = cache_len − pad_left[b]);
//   * the new token is appended to the cache by split 0 and folded into its online softmax from registers,
//     so the streamed range is [pad_left, cache_len) and nothing written in this launch is re-read;
//   * splits of the cache are chosen for the shape (see the dispatch), to cover load latency with parallelism;
//   * the last CTA of each (batch, kv-head) to finish — found with an atomic ticket — merges the partial
//     (m, l, o) triples, so there is no separate combine kernel.  The ticket counter is reset by that CTA.
// Reference semantics: jax_llama/model.py:201-300 at S = 1.
#include <atomic>

#include "common.cuh"
#include "tcgen05.cuh"
#include "jllama_b200.h"

namespace jl {

constexpr int DF_WARPS = 4;
constexpr int DF_KPI = 4;

struct FusedAttnParams {
  const __nv_bfloat16* qkv;      // [B, (nh + 2 nkv) · hd], not rotated
  __nv_bfloat16* kc;             // [B][nkv][T][hd]
  __nv_bfloat16* vc;
  const float* cos_t;            // [max_pos, hd/2]
  const float* sin_t;
  const int* cache_len_ptr;
  const int* pad_left;
  float* o_part;                 // [B·nh][splits][hd]
  float* ml_part;                // [B·nh][splits][2]
  int* tickets;                  // [B·nkv], zero on entry, zero on exit
  __nv_bfloat16* out;            // [B, nh·hd]
  int nkv, T, max_pos, splits;
  float scale_log2;
  int vec;                       // o_part on 16-byte and out on 8-byte boundaries
};

// Shared tail of both kernels: s_o / s_ml hold the (m, l, o) triples of the CTA's NG independent streams.  Folds them,
// then (splits > 1) the last CTA of this (batch, kv-head) to finish — found with an atomic ticket — merges the
// partial triples of all splits.  The ticket counter is reset by that CTA.
template <int NG, int G, int HD>
__device__ __forceinline__ void df_fold_and_merge(const FusedAttnParams& p, float (*s_o)[G][HD], float (*s_ml)[G][2],
                                                  int* s_last_p, const int b, const int kvh, const int split,
                                                  const int active) {
  const int nh = p.nkv * G;
  int& s_last = *s_last_p;
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * HD; idx += (int)blockDim.x) {
    const int g = idx / HD, d = idx - g * HD;
    float M = -INFINITY;
#pragma unroll
    for (int j = 0; j < NG; ++j) M = fmaxf(M, s_ml[j][g][0]);
    const float Ms = M == -INFINITY ? 0.f : M;
    float acc = 0.f, L = 0.f;
#pragma unroll
    for (int j = 0; j < NG; ++j) {
      const float w = exp2f(s_ml[j][g][0] - Ms);
      acc += w * s_o[j][g][d];
      L += w * s_ml[j][g][1];
    }
    const int h = kvh * G + g;
    if (active == 1) {
      p.out[((size_t)b * nh + h) * HD + d] = __float2bfloat16(L > 0.f ? acc / L : 0.f);
    } else {
      const size_t pi = ((size_t)b * nh + h) * p.splits + split;
      p.o_part[pi * HD + d] = acc;
      if (d == 0) { p.ml_part[pi * 2] = M; p.ml_part[pi * 2 + 1] = L; }
    }
  }
  if (active == 1) return;

  // ---- ticket: the last CTA of this (b, kv head) merges all splits
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    int* t = p.tickets + b * p.nkv + kvh;
    const int prev = atomicAdd(t, 1);
    s_last = prev == active - 1;
    if (s_last) *t = 0;                                  // everyone has arrived: safe to re-arm for the next launch
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // stage the (m, l) pairs of all splits in shared memory (one parallel round trip), then every thread
  // folds its outputs with independent, unrolled loads
  float* s_m = &s_o[0][0][0];                       // reuse: G*splits floats each, far below NG*G*HD
  float* s_l = s_m + G * 64;
  __syncthreads();
  for (int i = threadIdx.x; i < G * active; i += (int)blockDim.x) {
    const int g = i / active, sp = i - g * active;
    const size_t bh = (size_t)b * nh + kvh * G + g;
    s_m[g * 64 + sp] = __ldcg(p.ml_part + (bh * p.splits + sp) * 2);
    s_l[g * 64 + sp] = __ldcg(p.ml_part + (bh * p.splits + sp) * 2 + 1);
  }
  __syncthreads();
  if (!p.vec) {                                     // scratch or output off those boundaries: one column per thread
    for (int idx = threadIdx.x; idx < G * HD; idx += (int)blockDim.x) {
      const int g = idx / HD, d = idx - g * HD;
      const size_t bh = (size_t)b * nh + kvh * G + g;
      float M = -INFINITY;
      for (int sp = 0; sp < active; ++sp) M = fmaxf(M, s_m[g * 64 + sp]);
      const float Ms = M == -INFINITY ? 0.f : M;
      float acc = 0.f, L = 0.f;
      for (int sp = 0; sp < active; ++sp) {
        const float w = exp2f(s_m[g * 64 + sp] - Ms);
        if (w > 0.f) acc += w * __ldcg(p.o_part + (bh * p.splits + sp) * HD + d);
        L += w * s_l[g * 64 + sp];
      }
      p.out[bh * HD + d] = __float2bfloat16(acc * (L > 0.f ? 1.f / L : 0.f));
    }
    return;
  }
  // four columns per thread, the partial rows of 16 splits requested before the first is used (one memory round trip
  // for up to 16 splits: a loop with a remainder took one per remaining split, 15.2 us at 12 splits against 12.1 at 8)
  for (int idx = threadIdx.x; idx < G * (HD / 4); idx += (int)blockDim.x) {
    const int g = idx / (HD / 4), d = 4 * (idx - g * (HD / 4));
    const size_t bh = (size_t)b * nh + kvh * G + g;
    float M = -INFINITY;
    for (int sp = 0; sp < active; ++sp) M = fmaxf(M, s_m[g * 64 + sp]);
    const float Ms = M == -INFINITY ? 0.f : M;
    float acc[4] = {0.f, 0.f, 0.f, 0.f}, L = 0.f;
    const float* op = p.o_part + bh * p.splits * HD + d;
    for (int sp0 = 0; sp0 < active; sp0 += 16) {
      float4 ov[16];
#pragma unroll
      for (int i = 0; i < 16; ++i)
        ov[i] = sp0 + i < active ? __ldcg(reinterpret_cast<const float4*>(op + (size_t)(sp0 + i) * HD)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (sp0 + i < active) {
          const float w = exp2f(s_m[g * 64 + sp0 + i] - Ms);
          if (w > 0.f) { acc[0] += w * ov[i].x; acc[1] += w * ov[i].y; acc[2] += w * ov[i].z; acc[3] += w * ov[i].w; }
          L += w * s_l[g * 64 + sp0 + i];
        }
      }
    }
    const float inv = L > 0.f ? 1.f / L : 0.f;
    *reinterpret_cast<uint2*>(p.out + bh * HD + d) = make_uint2(pack_bf16(acc[0] * inv, acc[1] * inv), pack_bf16(acc[2] * inv, acc[3] * inv));
  }
}

template <int G, int HD>
__global__ void __launch_bounds__(DF_WARPS * 32) decode_attn_fused_kernel(const FusedAttnParams p) {
  constexpr int LPK = HD / 8;
  constexpr int GPW = 32 / LPK;
  constexpr int NG = DF_WARPS * GPW;
  constexpr int KEYS_PER_ITER = NG * DF_KPI;
  __shared__ float s_o[NG][G][HD];
  __shared__ float s_ml[NG][G][2];
  __shared__ int s_last;

  pdl_wait();
  pdl_launch_dependents();

  const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const int nh = p.nkv * G;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lig = lane % LPK;
  const int gid = warp * GPW + lane / LPK;
  const int group_base = lane - lig;
  const int kidx = ((lig / (LPK / 2)) & 1) * 2 + ((lig / (LPK / 4)) & 1);

  int len = *p.cache_len_ptr;                          // slots already filled; the new token takes slot `len`
  len = len > p.T ? p.T : len;
  const int first = p.pad_left ? p.pad_left[b] : 0;
  const int valid = len - first > 0 ? len - first : 0;
  int pos = len - first;
  pos = pos < 0 ? 0 : (pos >= p.max_pos ? p.max_pos - 1 : pos);
  int chunk = (valid + p.splits - 1) / p.splits;
  chunk = ((chunk + KEYS_PER_ITER - 1) / KEYS_PER_ITER) * KEYS_PER_ITER;
  const int lo = first + split * chunk;
  const int hi = lo + chunk < len ? lo + chunk : len;

  // rotation factors of this lane's 4 pairs
  const float4 cs4 = __ldg(reinterpret_cast<const float4*>(p.cos_t) + (size_t)pos * LPK + lig);
  const float4 sn4 = __ldg(reinterpret_cast<const float4*>(p.sin_t) + (size_t)pos * LPK + lig);
  const float cs[4] = {cs4.x, cs4.y, cs4.z, cs4.w}, sn[4] = {sn4.x, sn4.y, sn4.z, sn4.w};
  const __nv_bfloat16* row = p.qkv + (size_t)b * (nh + 2 * p.nkv) * HD;

  float qf[G][8];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const uint4 a = *reinterpret_cast<const uint4*>(row + (size_t)(kvh * G + g) * HD + lig * 8);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float re = bf16_lo(aw[j]), im = bf16_hi(aw[j]);
      // round the rotated q to bf16 like the unfused path does, then fold the softmax scale in
      const uint32_t r = pack_bf16(re * cs[j] - im * sn[j], re * sn[j] + im * cs[j]);
      qf[g][2 * j] = bf16_lo(r) * p.scale_log2;
      qf[g][2 * j + 1] = bf16_hi(r) * p.scale_log2;
    }
  }
  float m[G], l[G], o[G][8];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    m[g] = -INFINITY;
    l[g] = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) o[g][e] = 0.f;
  }

  const size_t head_off = ((size_t)b * p.nkv + kvh) * (size_t)p.T * HD;
  const __nv_bfloat16* kbase = p.kc + head_off + lig * 8;
  const __nv_bfloat16* vbase = p.vc + head_off + lig * 8;

  // one online-softmax update with DF_KPI keys per lane-group (K/V rows already in registers)
  auto process = [&](const uint4 (&kr)[DF_KPI], const uint4 (&vr)[DF_KPI], const int key0) {
      float part[G][DF_KPI];
#pragma unroll
      for (int i = 0; i < DF_KPI; ++i) {
        const float kf[8] = {bf16_lo(kr[i].x), bf16_hi(kr[i].x), bf16_lo(kr[i].y), bf16_hi(kr[i].y),
                             bf16_lo(kr[i].z), bf16_hi(kr[i].z), bf16_lo(kr[i].w), bf16_hi(kr[i].w)};
#pragma unroll
        for (int g = 0; g < G; ++g) {
          float s = 0.f;
#pragma unroll
          for (int e = 0; e < 8; ++e) s = fmaf(qf[g][e], kf[e], s);
          part[g][i] = s;
        }
      }
      float pr[G][DF_KPI];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const bool up = (lig & (LPK / 2)) != 0;
        float k0 = up ? part[g][2] : part[g][0], k1 = up ? part[g][3] : part[g][1];
        const float s0 = up ? part[g][0] : part[g][2], s1 = up ? part[g][1] : part[g][3];
        k0 += __shfl_xor_sync(0xffffffffu, s0, LPK / 2);
        k1 += __shfl_xor_sync(0xffffffffu, s1, LPK / 2);
        const bool up2 = (lig & (LPK / 4)) != 0;
        float s = up2 ? k1 : k0;
        const float snd = up2 ? k0 : k1;
        s += __shfl_xor_sync(0xffffffffu, snd, LPK / 4);
#pragma unroll
        for (int off = LPK / 8; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (key0 + kidx >= hi) s = -INFINITY;
        float mx = fmaxf(s, __shfl_xor_sync(0xffffffffu, s, LPK / 2));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, LPK / 4));
        const float m_new = fmaxf(m[g], mx);
        const float m_safe = m_new == -INFINITY ? 0.f : m_new;
        const float corr = exp2f(m[g] - m_safe);
        const float pe = exp2f(s - m_safe);
        m[g] = m_new;
        float psum = 0.f;
#pragma unroll
        for (int i = 0; i < DF_KPI; ++i) {
          pr[g][i] = __shfl_sync(0xffffffffu, pe, group_base + (i >> 1) * (LPK / 2) + (i & 1) * (LPK / 4));
          psum += pr[g][i];
        }
        l[g] = l[g] * corr + psum;
#pragma unroll
        for (int e = 0; e < 8; ++e) o[g][e] *= corr;
      }
#pragma unroll
      for (int i = 0; i < DF_KPI; ++i) {
        const float vf[8] = {bf16_lo(vr[i].x), bf16_hi(vr[i].x), bf16_lo(vr[i].y), bf16_hi(vr[i].y),
                             bf16_lo(vr[i].z), bf16_hi(vr[i].z), bf16_lo(vr[i].w), bf16_hi(vr[i].w)};
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
          for (int e = 0; e < 8; ++e) o[g][e] = fmaf(pr[g][i], vf[e], o[g][e]);
      }
  };

  // UNR iterations' worth of K/V loads are issued back to back before any of them is consumed, so a
  // 64-key split is a single memory round trip (warp-uniform trip count; tails are predicated)
  constexpr int UNR = G <= 4 ? 2 : 1;
  for (int base = lo; base < hi; base += UNR * KEYS_PER_ITER) {
    uint4 kr[UNR][DF_KPI], vr[UNR][DF_KPI];
#pragma unroll
    for (int u = 0; u < UNR; ++u) {
      const int key0 = base + u * KEYS_PER_ITER + gid * DF_KPI;
#pragma unroll
      for (int i = 0; i < DF_KPI; ++i) {
        const bool ok = key0 + i < hi;
        kr[u][i] = ok ? ldg_stream(kbase + (size_t)(key0 + i) * HD) : make_uint4(0, 0, 0, 0);
        vr[u][i] = ok ? ldg_stream(vbase + (size_t)(key0 + i) * HD) : make_uint4(0, 0, 0, 0);
      }
    }
#pragma unroll
    for (int u = 0; u < UNR; ++u) process(kr[u], vr[u], base + u * KEYS_PER_ITER + gid * DF_KPI);
  }

  // ---- the new token: rotate k, append k and v to the cache, fold it in from registers (split 0, warp 0)
  if (split == 0 && warp == 0) {
    const uint4 ka = *reinterpret_cast<const uint4*>(row + (size_t)(nh + kvh) * HD + lig * 8);
    const uint4 va = *reinterpret_cast<const uint4*>(row + (size_t)(nh + p.nkv + kvh) * HD + lig * 8);
    const uint32_t kw[4] = {ka.x, ka.y, ka.z, ka.w};
    uint32_t kr4[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float re = bf16_lo(kw[j]), im = bf16_hi(kw[j]);
      kr4[j] = pack_bf16(re * cs[j] - im * sn[j], re * sn[j] + im * cs[j]);
    }
    if (gid == 0 && len < p.T) {
      *reinterpret_cast<uint4*>(p.kc + head_off + (size_t)len * HD + lig * 8) = make_uint4(kr4[0], kr4[1], kr4[2], kr4[3]);
      *reinterpret_cast<uint4*>(p.vc + head_off + (size_t)len * HD + lig * 8) = va;
    }
    const float kf[8] = {bf16_lo(kr4[0]), bf16_hi(kr4[0]), bf16_lo(kr4[1]), bf16_hi(kr4[1]),
                         bf16_lo(kr4[2]), bf16_hi(kr4[2]), bf16_lo(kr4[3]), bf16_hi(kr4[3])};
    const float vf[8] = {bf16_lo(va.x), bf16_hi(va.x), bf16_lo(va.y), bf16_hi(va.y),
                         bf16_lo(va.z), bf16_hi(va.z), bf16_lo(va.w), bf16_hi(va.w)};
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float s = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) s = fmaf(qf[g][e], kf[e], s);
#pragma unroll
      for (int off = LPK / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      if (gid != 0) s = -INFINITY;                       // counted once, by lane-group 0
      const float m_new = fmaxf(m[g], s);
      const float m_safe = m_new == -INFINITY ? 0.f : m_new;
      const float corr = exp2f(m[g] - m_safe);
      const float pe = exp2f(s - m_safe);
      m[g] = m_new;
      l[g] = l[g] * corr + pe;
#pragma unroll
      for (int e = 0; e < 8; ++e) o[g][e] = o[g][e] * corr + pe * vf[e];
    }
  }

  // ---- fold the lane-groups of this CTA
#pragma unroll
  for (int g = 0; g < G; ++g) {
#pragma unroll
    for (int e = 0; e < 8; ++e) s_o[gid][g][lig * 8 + e] = o[g][e];
    if (lig == 0) { s_ml[gid][g][0] = m[g]; s_ml[gid][g][1] = l[g]; }
  }
  df_fold_and_merge<NG, G, HD>(p, s_o, s_ml, &s_last, b, kvh, split, p.splits);
}

// =====================================================================================================================
// Tensor-core variant (the shapes that take it: rule at the dispatch below).
//
// Why: at batch 32 / 2k context the kernel above moves 268 MB per layer in 133 µs (2 TB/s) — ncu shows ~1 issued
// instruction per cycle and no memory stall: the bf16 → fp32 unpacking and the G x 256 FMAs per key are the limit,
// not HBM.  Here both products go through mma.sync.m16n8k16 (bf16 in, fp32 accumulate) with the G query heads of
// the kv head as rows 0..G-1 of the 16-row operand.
//   * Every warp is a stream of its own: one lane keeps DM_STAGES blocks of KPI keys (K and V, 128-byte swizzled TMA
//     boxes) in flight into the warp's ring in shared memory, the warp reads them with ldmatrix and runs its own online
//     softmax.  No barrier between warps until the fold.  Keeping the blocks in registers instead (fragments loaded
//     from an L2 prefetched two blocks ahead) left one memory round trip exposed per block:
//     24 rows x 8 heads, 3500 keys, 80 us (4.6 TB/s) before and 64 (5.7) with the rings, 16 x 8 heads 18.4 and 13.9.
//   * P goes into the second product as high + low bfloat16 parts, in the two halves of the 16-row operand: rows
//     0..7 hold the high parts and rows 8..15 the low ones, so that 16 bits of P cost no instruction more than 8 would;
//     the two halves of the accumulator are added at the end.
//     Against float64 (2-norm of the bfloat16 result; fp32 P in the SIMT kernel -> this one): 1 x 8 heads of 128, 4000 keys 1.64430e-3 ->
//     1.64430e-3; 16 x 8 heads of 64, 2500 keys 1.65879e-3 -> 1.65879e-3; two results of a thousand round the other way.
// The new token is folded in by the same code as a block whose only valid key is slot 0.  One CTA alone runs at the latency of
// its dependent steps (ldmatrix → S → maximum → exponentials → P·V, ~0.6 us per 16 keys of a warp), many at HBM's rate.
constexpr int DM_WARPS = 4;
constexpr int DM_STAGES = 3;
template <int HD> struct DmTile {
  static constexpr int KPI = HD == 128 ? 16 : 32;            // keys of a block: 8 KB of K and V at either width
  static constexpr int ONE_SPLIT = 40960 / HD;               // keys that one CTA takes rather than split (320, 640)
  static constexpr int HALVES = HD / 64;                     // 64-column boxes of a row
  static constexpr int BOX = KPI * 128;                      // bytes
  static constexpr int STAGE = 2 * HALVES * BOX;
  static constexpr int SMEM = DM_WARPS * DM_STAGES * STAGE + 1024;
};

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void dm_ldsm(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void dm_ldsm_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// rotate the four (re, im) pairs of one 16-byte chunk; pair j uses cos/sin entry j of cs / sn
__device__ __forceinline__ uint4 rope_chunk(const uint4 a, const float4 cs, const float4 sn) {
  const uint32_t w[4] = {a.x, a.y, a.z, a.w};
  const float c[4] = {cs.x, cs.y, cs.z, cs.w}, s[4] = {sn.x, sn.y, sn.z, sn.w};
  uint32_t r[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float re = bf16_lo(w[j]), im = bf16_hi(w[j]);
    r[j] = pack_bf16(re * c[j] - im * s[j], re * s[j] + im * c[j]);
  }
  return make_uint4(r[0], r[1], r[2], r[3]);
}

template <int G, int HD>
__global__ void __launch_bounds__(DM_WARPS * 32, 2)
    decode_attn_mma_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const FusedAttnParams p) {
  using Tile = DmTile<HD>;
  constexpr int KPI = Tile::KPI, HALVES = Tile::HALVES;
  constexpr int NT = KPI / 8;                  // 8-key S tiles per block
  constexpr int NB = KPI / 16;                 // 16-key P·V steps per block
  constexpr int KS = HD / 16;                  // k-steps of S
  extern __shared__ uint8_t dm_smem[];
  __shared__ float s_ml[DM_WARPS][G][2];
  __shared__ __align__(8) uint64_t s_bar[DM_WARPS][DM_STAGES];
  __shared__ int s_last;
  static_assert(DM_WARPS * G * HD * 4 <= Tile::SMEM - 1024, "the partial outputs take the ring's place");

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const uint32_t raw = tc::smem_u32(dm_smem);
  const uint32_t ring0 = (raw + 1023u) & ~1023u;
  const uint32_t ring = ring0 + warp * (DM_STAGES * Tile::STAGE);
  const uint32_t bar0 = tc::smem_u32(&s_bar[warp][0]);
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < DM_STAGES; ++i) tc::mbar_init(bar0 + 8 * i, 1);
    tc::fence_barrier_init();
  }
  __syncwarp();

  pdl_wait();
  pdl_launch_dependents();

  const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const int nh = p.nkv * G;

  int len = *p.cache_len_ptr;
  len = len > p.T ? p.T : len;
  const int first = p.pad_left ? p.pad_left[b] : 0;
  const int valid = len - first > 0 ? len - first : 0;
  int pos = len - first;
  pos = pos < 0 ? 0 : (pos >= p.max_pos ? p.max_pos - 1 : pos);
  int chunk = (valid + p.splits - 1) / p.splits;
  chunk = ((chunk + DM_WARPS * KPI - 1) / (DM_WARPS * KPI)) * (DM_WARPS * KPI);
  if (valid <= Tile::ONE_SPLIT) chunk = valid;            // the merge would cost more than the keys
  const int active = valid > 0 ? (valid + chunk - 1) / chunk : 1;
  if (split >= active) return;
  const int lo = first + split * chunk;
  const int hi = lo + chunk < len ? lo + chunk : len;

  const int row0 = (b * p.nkv + kvh) * p.T;              // first cache row of this head in the [B·nkv·T, HD] view
  // one lane asks for a block; a box may run past the last key (next head's rows, or zeros past the cache): those keys
  // are masked below
  auto request = [&](const int base, const int st) {
    if (lane == 0 && base < hi) {
      const uint32_t dst = ring + st * Tile::STAGE, bar = bar0 + 8 * st;
      tc::mbar_expect_tx(bar, Tile::STAGE);
#pragma unroll
      for (int h = 0; h < HALVES; ++h) {
        tc::tma_load_2d(dst + h * Tile::BOX, &tm_k, bar, 64 * h, row0 + base, tc::EVICT_FIRST);
        tc::tma_load_2d(dst + (HALVES + h) * Tile::BOX, &tm_v, bar, 64 * h, row0 + base, tc::EVICT_FIRST);
      }
    }
  };
#pragma unroll
  for (int i = 0; i < DM_STAGES; ++i) request(lo + (i * DM_WARPS + warp) * KPI, i);

  // the new token belongs to the last warp of the last working split, which has the fewest keys
  const bool newest = split == active - 1 && warp == DM_WARPS - 1;
  const __nv_bfloat16* row = p.qkv + (size_t)b * (nh + 2 * p.nkv) * HD;
  uint4 kn = make_uint4(0, 0, 0, 0), vn = kn;             // chunk `lane` of its rows, asked for ahead of the loop
  if (newest && lane < HD / 8) {
    kn = *reinterpret_cast<const uint4*>(row + (size_t)(nh + kvh) * HD + 8 * lane);
    vn = *reinterpret_cast<const uint4*>(row + (size_t)(nh + p.nkv + kvh) * HD + 8 * lane);
  }
  const float* cos_p = p.cos_t + (size_t)pos * (HD / 2);
  const float* sin_p = p.sin_t + (size_t)pos * (HD / 2);

  // Q of head kvh·G + g, rotated and rounded to bf16 (as the unfused path does): qa[s] = (a0, a2) of k-step s
  uint32_t qa[KS][2];
#pragma unroll
  for (int s = 0; s < KS; ++s)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      qa[s][i] = 0;
      if (g < G) {
        const int pair = 8 * s + 4 * i + t;
        const uint32_t w = *reinterpret_cast<const uint32_t*>(row + (size_t)(kvh * G + g) * HD + 2 * pair);
        const float c = __ldg(cos_p + pair), sn = __ldg(sin_p + pair), re = bf16_lo(w), im = bf16_hi(w);
        qa[s][i] = pack_bf16(re * c - im * sn, re * sn + im * c);
      }
    }

  float m = -INFINITY, l = 0.f;                // row g: m is quad-uniform, l is this thread's share of the sum
  float o[HD / 8][4];                          // [0..1]: row g against P's high parts, [2..3]: against the low parts
#pragma unroll
  for (int e = 0; e < HD / 8; ++e)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[e][i] = 0.f;

  // ldmatrix addresses within a 64-column box: row r's 16-byte chunk c lies at r * 128 + ((c ^ (r & 7)) << 4)
  const int l7 = lane & 7, q8 = lane >> 3;
  uint32_t koff[2], voff[4];
#pragma unroll
  for (int i = 0; i < 2; ++i) koff[i] = l7 * 128 + (((4 * i + q8) ^ l7) << 4);
#pragma unroll
  for (int i = 0; i < 4; ++i) voff[i] = ((q8 & 1) * 8 + l7) * 128 + (((2 * i + (q8 >> 1)) ^ l7) << 4);

  // one online-softmax update with the block in stage `st`; keys >= limit are masked
  auto process = [&](const int st, const int base, const int limit) {
    const uint32_t ks = ring + st * Tile::STAGE, vs = ks + HALVES * Tile::BOX;
    float c[NT][2];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      float d[2][4] = {};                                  // two chains: half the latency of the dependent products
#pragma unroll
      for (int i = 0; i < KS / 2; ++i) {
        uint32_t r[4];
        dm_ldsm(ks + (i >> 1) * Tile::BOX + j * 1024 + koff[i & 1], r);
        mma_16816(d[0], qa[2 * i][0], 0u, qa[2 * i][1], 0u, r[0], r[1]);
        mma_16816(d[1], qa[2 * i + 1][0], 0u, qa[2 * i + 1][1], 0u, r[2], r[3]);
      }
      c[j][0] = d[0][0] + d[1][0];
      c[j][1] = d[0][1] + d[1][1];
    }
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int key = base + 8 * j + 2 * t;
      c[j][0] = key < limit ? c[j][0] * p.scale_log2 : -INFINITY;
      c[j][1] = key + 1 < limit ? c[j][1] * p.scale_log2 : -INFINITY;
      mx = fmaxf(mx, fmaxf(c[j][0], c[j][1]));
    }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float m_new = fmaxf(m, mx);
    const float m_safe = m_new == -INFINITY ? 0.f : m_new;
    const float corr = exp2f(m - m_safe);
    m = m_new;
    float psum = 0.f;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      c[j][0] = exp2f(c[j][0] - m_safe);
      c[j][1] = exp2f(c[j][1] - m_safe);
      psum += c[j][0] + c[j][1];
    }
    l = l * corr + psum;
    if (__any_sync(0xffffffffu, corr != 1.f)) {
#pragma unroll
      for (int e = 0; e < HD / 8; ++e)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[e][i] *= corr;
    }
#pragma unroll
    for (int kb = 0; kb < NB; ++kb) {
      const float(&c0)[2] = c[2 * kb];
      const float(&c1)[2] = c[2 * kb + 1];
      const uint32_t h0 = pack_bf16(c0[0], c0[1]), h2 = pack_bf16(c1[0], c1[1]);
      const uint32_t l0 = pack_bf16(c0[0] - bf16_lo(h0), c0[1] - bf16_hi(h0));
      const uint32_t l2 = pack_bf16(c1[0] - bf16_lo(h2), c1[1] - bf16_hi(h2));
#pragma unroll
      for (int e = 0; e < HD / 16; ++e) {
        uint32_t r[4];
        dm_ldsm_t(vs + (e >> 2) * Tile::BOX + kb * 2048 + voff[e & 3], r);
        mma_16816(o[2 * e], h0, l0, h2, l2, r[0], r[1]);
        mma_16816(o[2 * e + 1], h0, l0, h2, l2, r[2], r[3]);
      }
    }
  };
  // V rows [n, KPI) of a stage hold no key: zero them, a weight of zero times an unused slot's NaN would be NaN
  auto zero_v_rows = [&](const int st, const int n) {
    for (int i = lane; i < (KPI - n) * 8 * HALVES; i += 32) {
      const int r = n + i / (8 * HALVES), c = i % (8 * HALVES);
      const uint32_t a = ring + st * Tile::STAGE + (HALVES + (c >> 3)) * Tile::BOX + r * 128 + (c & 7) * 16;
      asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(a), "r"(0) : "memory");
    }
    __syncwarp();
  };

  int st = 0;
  uint32_t phase = 0;
  for (int base = lo + warp * KPI; base < hi; base += DM_WARPS * KPI) {
    tc::mbar_wait(bar0 + 8 * st, phase);
    if (base + KPI > hi) zero_v_rows(st, hi - base);
    process(st, base, hi);
    __syncwarp();                                          // every lane has read the stage: it may be filled again
    request(base + DM_STAGES * DM_WARPS * KPI, st);
    if (++st == DM_STAGES) { st = 0; phase ^= 1; }
  }

  // ---- the new token: rotate k, append k and v to the cache, fold it in as key 0 of a block
  if (newest) {                                            // all copies into this warp's ring have been waited for
    const size_t slot = ((size_t)row0 + len) * HD;
    if (lane < HD / 8) {                                   // row 0 of a box is not permuted
      kn = rope_chunk(kn, __ldg(reinterpret_cast<const float4*>(cos_p) + lane), __ldg(reinterpret_cast<const float4*>(sin_p) + lane));
      if (len < p.T) {
        *reinterpret_cast<uint4*>(p.kc + slot + 8 * lane) = kn;
        *reinterpret_cast<uint4*>(p.vc + slot + 8 * lane) = vn;
      }
      const uint32_t a = ring + (lane >> 3) * Tile::BOX + (lane & 7) * 16;
      asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(kn.x), "r"(kn.y), "r"(kn.z), "r"(kn.w) : "memory");
      asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a + HALVES * Tile::BOX), "r"(vn.x), "r"(vn.y), "r"(vn.z), "r"(vn.w)
                   : "memory");
    }
    zero_v_rows(0, 1);
    process(0, 0, 1);
  }

  // ---- this warp's triple → shared memory, over the rings once every warp is done with its own
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  __syncthreads();
  float(*s_o)[G][HD] = reinterpret_cast<float(*)[G][HD]>(dm_smem + (ring0 - raw));
  if (g < G) {
#pragma unroll
    for (int e = 0; e < HD / 8; ++e)
      *reinterpret_cast<float2*>(&s_o[warp][g][8 * e + 2 * t]) = make_float2(o[e][0] + o[e][2], o[e][1] + o[e][3]);
    if (t == 0) { s_ml[warp][g][0] = m; s_ml[warp][g][1] = l; }
  }
  df_fold_and_merge<DM_WARPS, G, HD>(p, s_o, s_ml, &s_last, b, kvh, split, active);
}

template <int G, int HD>
static int launch_decode_mma(const FusedAttnParams& p, int B, cudaStream_t s) {
  CUtensorMap tk, tv;
  const uint64_t rows = (uint64_t)B * p.nkv * p.T;
  int rc = make_tmap_2d_bf16(&tk, p.kc, rows, HD, HD, DmTile<HD>::KPI);
  if (rc == JL_OK) rc = make_tmap_2d_bf16(&tv, p.vc, rows, HD, HD, DmTile<HD>::KPI);
  if (rc != JL_OK) return rc;
  // attributes belong to the device's context: set at the first call on each (bit per device; setting them twice is harmless)
  static std::atomic<uint64_t> set{0};
  int dev = 0;
  JL_CUDA(cudaGetDevice(&dev));
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (bit == 0 || !(set.load(std::memory_order_acquire) & bit)) {
    JL_CUDA(cudaFuncSetAttribute(decode_attn_mma_kernel<G, HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, DmTile<HD>::SMEM));
    JL_CUDA(cudaFuncSetAttribute(decode_attn_mma_kernel<G, HD>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    set.fetch_or(bit, std::memory_order_release);
  }
  JL_CUDA(launch_pdl(decode_attn_mma_kernel<G, HD>, dim3(p.splits, p.nkv, B), dim3(DM_WARPS * 32), DmTile<HD>::SMEM, s, tk, tv, p));
  return JL_OK;
}

}  // namespace jl

using namespace jl;

static int g_attn_variant = 0;      // 0 = by shape, 1 = SIMT kernel, 2 = tensor-core kernel

// Pins the kernel behind jl_decode_attn_fused (tests and A/B measurements); 0 restores the shape-based choice.
extern "C" JL_API int jl_decode_attn_fused_set_variant(int variant) {
  JL_CHECK_ARG(variant >= 0 && variant <= 2, "jl_decode_attn_fused_set_variant: %d outside 0..2", variant);
  g_attn_variant = variant;
  return JL_OK;
}

extern "C" JL_API size_t jl_decode_attn_fused_scratch_bytes(int B, int nh, int nkv, int hd, int splits) {
  const size_t parts = splits <= 1 ? 0 : (size_t)B * nh * splits * (hd + 2) * sizeof(float);
  return parts + (size_t)B * nkv * sizeof(int);
}

extern "C" JL_API int jl_decode_attn_fused_splits(int B, int nkv, int max_len, int num_sms) {
  if (num_sms <= 0) num_sms = 148;
  int want = (4 * num_sms + B * nkv - 1) / (B * nkv);
  const int cap = (max_len + 127) / 128;                 // at least 128 keys per split
  int s = want < cap ? want : cap;
  return s < 1 ? 1 : (s > 64 ? 64 : s);
}

extern "C" JL_API int jl_decode_attn_fused(const void* qkv, void* k_cache, void* v_cache, const float* cos_t,
                                           const float* sin_t, const int* cache_len_ptr, const int* pad_left,
                                           void* scratch, void* out, int B, int nh, int nkv, int hd, int T,
                                           int max_pos, float scale, int splits, void* stream) {
  JL_CHECK_ARG(nkv > 0 && nh % nkv == 0, "jl_decode_attn_fused: nh=%d not a multiple of nkv=%d", nh, nkv);
  JL_CHECK_ARG(splits >= 1 && splits <= 64, "jl_decode_attn_fused: splits=%d outside 1..64", splits);
  JL_CHECK_ARG(scratch != nullptr && cache_len_ptr != nullptr, "jl_decode_attn_fused: scratch and cache_len are required");
  if (B == 0) return JL_OK;
  const int G = nh / nkv;
  FusedAttnParams p{};
  p.qkv = (const __nv_bfloat16*)qkv; p.kc = (__nv_bfloat16*)k_cache; p.vc = (__nv_bfloat16*)v_cache;
  p.cos_t = cos_t; p.sin_t = sin_t; p.cache_len_ptr = cache_len_ptr; p.pad_left = pad_left;
  const size_t part_floats = splits <= 1 ? 0 : (size_t)B * nh * splits * hd;
  p.o_part = (float*)scratch;
  p.ml_part = p.o_part + part_floats;
  p.tickets = (int*)(p.ml_part + (splits <= 1 ? 0 : (size_t)B * nh * splits * 2));
  p.out = (__nv_bfloat16*)out;
  p.nkv = nkv; p.T = T; p.max_pos = max_pos; p.splits = splits;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.vec = (uintptr_t)scratch % 16 == 0 && (uintptr_t)out % 8 == 0;
  auto s = (cudaStream_t)stream;
  cudaError_t e = cudaErrorInvalidValue;
  // The tensor-core kernel, but for one query head per kv head over a cache of at most 128 slots, where the ring and the 16-row products have
  // nothing to share and the SIMT kernel's shorter start wins (SIMT and this one, us in a graph: 4 heads of 128, 128 slots 2.8 and 3.7, of 64
  // 2.3 and 2.8; at 160 slots 5.3 and 3.7, 4.9 and 2.9).  Everywhere else it is the faster one: 3 x 4 heads of 64, 100 keys, two query heads
  // each 3.1 and 2.8, four 3.4 and 3.0; 1 x 8 heads, 4000 keys 20 and 9.1; 16 x 8 heads of 64, 2500 keys 52 and 15.7; 24 x 8 heads, 4000 keys 193
  // and 64.
  const bool use_mma = (hd == 128 || hd == 64) && (g_attn_variant == 2 || (g_attn_variant == 0 && !(G == 1 && T <= 128)));
  if (use_mma) {
    static int sms = 0;
    if (sms == 0) {
      int dev = 0;
      if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        sms = 148;
    }
    // Splits by estimate, the caller's count (which sizes the scratch) being the most there may be.  A call costs the
    // larger of its bytes and of the waves of CTAs (2 per SM) times the keys of one CTA at the pace of its dependent
    // blocks; each wave adds the way from the position to the first block, splitting adds the merge.  The five constants are
    // fits to 31 shapes swept over 1 to 32 splits; the choice was within 5 % of the best count in all but two of them (8 %).
    const int slots = 2 * sms, pairs = B * nkv, step = hd == 128 ? 64 : 128;
    const float key_us = hd == 128 ? 0.0091f : 0.0039f, bw_us = (float)pairs * (float)T * (float)hd * 4.f / 6.0e6f;
    int ms = 1;
    float best = 0.f;
    for (int c = 1; c <= splits && c <= 32; ++c) {
      const float waves = (float)((pairs * c + slots - 1) / slots);
      const float chunk = (float)(((T + c - 1) / c + step - 1) / step * step);
      const float us = fmaxf(bw_us, waves * chunk * key_us) + 3.4f * waves + (c > 1 ? 2.5f + 0.12f * c : 0.f);
      if (c == 1 || us < best) { best = us; ms = c; }
    }
    p.splits = ms;
#define JL_DM(G_, HD_) if (G == G_ && hd == HD_) return launch_decode_mma<G_, HD_>(p, B, s);
    JL_DM(1, 128) JL_DM(2, 128) JL_DM(4, 128) JL_DM(8, 128)
    JL_DM(1, 64) JL_DM(2, 64) JL_DM(4, 64) JL_DM(8, 64)
#undef JL_DM
  }
#define JL_DF(G_, HD_) \
  if (G == G_ && hd == HD_) e = launch_pdl(decode_attn_fused_kernel<G_, HD_>, dim3(splits, nkv, B), dim3(DF_WARPS * 32), 0, s, p);
  JL_DF(1, 128) else JL_DF(2, 128) else JL_DF(4, 128) else JL_DF(8, 128)
  else JL_DF(1, 64) else JL_DF(2, 64) else JL_DF(4, 64) else JL_DF(8, 64)
  else {
    set_error("jl_decode_attn_fused: unsupported GQA group %d / head_dim %d (groups 1,2,4,8; head_dim 64,128)", G, hd);
    return JL_ERR_UNSUPPORTED;
  }
#undef JL_DF
  JL_CUDA(e);
  return JL_OK;
}

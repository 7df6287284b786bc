// What the kernels of the linear recurrences share: parameters, and the values of a token and channel (gla_scan.cu, gla_chunk.cu).
#pragma once
#include "common.cuh"
#include "seq_types.cuh"

namespace jl {

__device__ __forceinline__ float log_sigmoid(float z) {
  return fminf(z, 0.0f) - log1pf(expf(-fabsf(z)));           // (no branch: lanes of either sign took both sides one after the other)
}

struct GlaParams {
  const float* y; int ldy;
  int q_off, k_off, v_off, a_off;      // columns of y: q [H*D], k [H*D], v [H*Dv], low-rank decay input [R]
  int B, S, H, D, Dv, R, P;
  float q_scale, inv_tau;
  const int* cache_len; const int* pad_left;
  float* state;                        // [B][H][D][Dv] fp32, read and written
  float* o;                            // [B*S][H][Dv] fp32
  // time chunks of the prompt scan (gla_stream_kernel): NC chunks of L tokens per row
  int NC, L;
  float* cstate;                       // [B][NC][H][D][Dv]: local end states (after mode 1), incoming states (after the combine)
  float* cdecay;                       // [B][NC][H][D]: product of the chunk's decays per key channel
  // retention (jl_retention_scan): one fixed decay per head instead of the projected one, rotary embedding of q and k at the
  // token's position, k scaled after the rotation
  const float* head_decay;             // [H] fp32, or nullptr: alpha from the low-rank projection
  const float* cos_t; const float* sin_t; int rot, layout, max_pos;      // tables [max_pos][rot/2]; rot == 0: no rotation
  float k_scale;
  // state space scan (jl_ssd_scan): q / k are shared by the qk_div heads of a group; the decay of (token, head) is
  // aux[m * ld_aux + h] and the value row is scaled by aux[m * ld_aux + H + h]
  int qk_div;                          // heads per q / k head (1: every head has its own)
  const float* aux; int ld_aux;
  // linear attention over activated projections: q, k and v pass `act` (ACT_NONE: as they are)
  int act;
  // matrix memory (jl_mlstm_scan): the last `ones` (0 or 1) of the Dv columns are not in y but constantly one before the value
  // scale, so the state's last column is the normaliser n and the last read-out column n . q
  int ones;
};

__device__ __forceinline__ float scan_value(const GlaParams& p, size_t m, int h, int c) {
  if (c >= p.Dv) return 0.0f;
  const int dv = p.Dv - p.ones;
  float v = c < dv ? p.y[m * p.ldy + p.v_off + h * dv + c] : 1.0f;
  if (p.act != ACT_NONE) v = apply_act(v, p.act, 0.0f, 0.0f);
  return p.aux ? v * p.aux[m * p.ld_aux + p.H + h] : v;
}

// q and k of channel d of head h for the token whose projection row is y[m] (position pos).
__device__ __forceinline__ void scan_qk(const GlaParams& p, size_t m, int h, int d, int pos, float& qv, float& kv) {
  const float* yr = p.y + m * p.ldy;
  const int hq = p.qk_div > 1 ? h / p.qk_div : h;
  const float* qh = yr + p.q_off + hq * p.D;
  const float* kh = yr + p.k_off + hq * p.D;
  if (p.rot > 0) {
    const float* ct = p.cos_t + (size_t)pos * (p.rot / 2);
    const float* st = p.sin_t + (size_t)pos * (p.rot / 2);
    qv = rotary_channel(qh, d, p.rot, p.layout, ct, st) * p.q_scale;
    kv = rotary_channel(kh, d, p.rot, p.layout, ct, st) * p.k_scale;
  } else if (p.act != ACT_NONE) {
    qv = apply_act(qh[d], p.act, 0.0f, 0.0f) * p.q_scale;
    kv = apply_act(kh[d], p.act, 0.0f, 0.0f) * p.k_scale;
  } else {
    qv = qh[d] * p.q_scale;
    kv = kh[d] * p.k_scale;
  }
}

// q, k and alpha; zs: the token's low-rank decay input
template <typename T>
__device__ __forceinline__ void scan_channel(const GlaParams& p, size_t m, int h, int d, int pos,
                                             const float* __restrict__ zs, const T* __restrict__ a2, const T* __restrict__ a2b,
                                             float& qv, float& kv, float& av) {
  scan_qk(p, m, h, d, pos, qv, kv);
  if (p.aux) { av = p.aux[m * p.ld_aux + h]; return; }
  if (p.head_decay) { av = p.head_decay[h]; return; }
  const int n = h * p.D + d;
  float z = to_f(a2b[n]);
  for (int r = 0; r < p.R; ++r) z = fmaf(to_f(a2[(size_t)n * p.R + r]), zs[r], z);
  av = expf(log_sigmoid(z) * p.inv_tau);
}

__device__ __forceinline__ int scan_position(const GlaParams& p, int b, int s) {
  if (p.rot <= 0) return 0;
  const int pos = (p.cache_len ? *p.cache_len : 0) + s - (p.pad_left ? p.pad_left[b] : 0);
  return pos < 0 ? 0 : (pos >= p.max_pos ? p.max_pos - 1 : pos);
}

// Prompts in chunks of 64 tokens (gla_chunk.cu): whether it takes these sizes, the floats of its workspace, and the launch (a JL_ code).
bool gla_chunk_takes(int B, int S, int H, int D, int Dv);
size_t gla_chunk_ws_floats(int B, int S, int H, int D, int Dv);
int gla_chunk_launch(GlaParams p, const void* a2, const void* a2_bias, float* ws, int dtype, cudaStream_t st);

__global__ void gla_combine_kernel(GlaParams p);

}  // namespace jl

// Host interface of the tcgen05 prompt attention for the head shapes of the generic attention kernels (flash_wide.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace jl {

struct FlashWide {
  __nv_bfloat16* out;               // [B, S, H, Dv]
  const int* cache_len;             // slots filled before this call's tokens (device scalar), or nullptr = 0
  const int* pad_left;              // [B] or nullptr
  int B, S, H, G;
  float scale_log2;                 // score scale · log2(e)
  int window, chunk;                // as in the generic kernels: > 0 limits the keys a query sees
  int sink; const float* sink_logit;
  const float* gate; int ldg;       // fp32 pre-activation of a sigmoid per (token, head), or nullptr
};

// whether the kernel takes these sizes, pitches and addresses (bfloat16 operands, no capped scores, no rotated values, no gate per channel)
bool flash_wide_takes(int S, int D, int Dv, int T_cap, int ldk, int ldv, long long k_bs, long long k_hs, long long v_bs, long long v_hs,
                      const void* q, const void* k, const void* v, const void* out);
int flash_wide_launch(const FlashWide& p, int D, int Dv, int T_cap, int ldk, int ldv, long long k_bs, long long k_hs, long long v_bs,
                      long long v_hs, const void* q, const void* k, const void* v, cudaStream_t st);

}  // namespace jl

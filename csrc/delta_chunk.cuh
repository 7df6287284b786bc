// Host interface of the delta rule with one decay per head over prompts, in chunks (delta_chunk.cu).
#pragma once
#include <cuda_runtime.h>

namespace jl {

struct DeltaHeadParams {
  const float* u; int ldu;           // q | k | v after their convolutions
  int q_off, k_off, v_off, G;        // G q / k heads shared by H / G heads each
  const float* y; int ldy;           // projection row: beta logits and decay inputs, one of each per head
  int b_off, a_off;
  int B, S, H, D, Dv, P, cols;
  const int* cache_len; const int* pad_left;
  float* state; float* o;
  float* qk; float* pair; float* gate; float* val;       // workspace parts (the walk token by token)
};

__device__ __forceinline__ float delta_softplus(float z) { return z > 20.0f ? z : log1pf(expf(z)); }
__device__ __forceinline__ float delta_head_decay(float z, float a_log) { return expf(-expf(a_log) * delta_softplus(z)); }

// whether keys of D channels are taken; floats of workspace; both launches
bool delta_chunk_takes(int D);
size_t delta_chunk_ws_floats(int B, int S, int H, int D);
int delta_chunk_launch(const DeltaHeadParams& p, float* ws, const void* a_bias, const void* a_log, int dtype, cudaStream_t st);

}  // namespace jl

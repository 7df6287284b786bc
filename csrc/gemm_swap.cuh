// Host interface of the few-token GEMM (gemm_swap.cu).
#pragma once
#include <cuda_runtime.h>

namespace jl {

enum { SWAP_PLAIN = 0, SWAP_RESIDUAL = 1, SWAP_SWIGLU = 2 };

// whether the kernel is the one for these sizes
bool gemm_swap_takes(int M, int N, int K, int num_sms, bool aligned);
// out = x [M, K] · w [N, K]^T for M <= 256, N % 8 == 0, K % 8 == 0 (modes as in jl_gemm)
int gemm_swap(const void* x, const void* w, const void* residual, void* out, int M, int N, int K, int mode, bool out_f32, int num_sms,
              unsigned long long* trace, cudaStream_t stream);
// out fp32 [M, N] for few output features (N <= 64) and many tokens
bool gemm_turned_takes(int M, int N, int K, int num_sms, bool aligned);
int gemm_turned_f32(const void* x, const void* w, void* out, int M, int N, int K, int num_sms, unsigned long long* trace, cudaStream_t s);
// whether K may be split over the CTAs of a cluster on a device
void gemm_swap_allow_split(int device, bool on);

}  // namespace jl

// What the float32 linears on tensor cores share (linear_f32.cu, linear_f32_pair.cu), and the host interface of the first.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

namespace jl {

// Many small products in one launch.  Plain batches: batch z reads x + (z / x_div) * x_bs, weights
// w + (w_index ? w_index[z] : z) * w_bs (w_index[z] < 0: the batch is skipped) and writes out + z * o_bs (per-head matrices; one expert per (token, choice) pair when
// decoding a mixture of experts: x_div = choices per token, so that the pairs of a token read the same input row).
// Sorted rows (tiled kernels only): the rows come in tiles of LT_BM that each belong to one weight matrix, tile_group[tile]
// (< 0: empty tile); row position p reads input row row_src[p] (< 0: padding, read as zero; nullptr: p itself) and writes
// output row p — the prompt path of a mixture of experts after its tokens were sorted by expert.
struct LinearGroup {
  long long x_bs, w_bs, o_bs;
  int x_div;
  const int* w_index;
  const int* tile_group;
  const int* row_src;
};

constexpr int LT_BM = 64;           // rows of a sorted tile

// eight consecutive floats -> the 16 bytes of each part
__device__ __forceinline__ void lf_split8(const float4& a, const float4& b, uint4 (&part)[3]) {
  const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  uint32_t h[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float r0 = v[2 * i], r1 = v[2 * i + 1];
    h[0][i] = pack_bf16(r0, r1);
    r0 -= bf16_lo(h[0][i]);
    r1 -= bf16_hi(h[0][i]);
    h[1][i] = pack_bf16(r0, r1);
    h[2][i] = pack_bf16(r0 - bf16_lo(h[1][i]), r1 - bf16_hi(h[1][i]));            // at most 8 significant bits: exact
  }
#pragma unroll
  for (int p = 0; p < 3; ++p) part[p] = make_uint4(h[p][0], h[p][1], h[p][2], h[p][3]);
}

// whether the tensor-core kernel takes these sizes, pitches and addresses
bool linear_f32_takes(int M, int K, int ldx, const LinearGroup& g, const void* x, const void* w);
// how it takes a plain product of these sizes: rows per tile, CTAs that share one, sums of 64 k that each of them adds in a row, tiles
struct LinearF32Plan { int bn, splits, chain; long tiles; };
LinearF32Plan linear_f32_plan(int M, int N, int K);
cudaError_t linear_f32_launch(const float* x, int ldx, const float* w, float* out, int ldo, int M, int N, int K, int act, float p0, float p1,
                              cudaStream_t st, const LinearGroup& g, int nbatch);

}  // namespace jl

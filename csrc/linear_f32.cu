// float32 linears of more than a few rows on tcgen05 tensor cores, with the accuracy of fp32 FMAs.  (Many rows over enough features: linear_f32_pair.cu; batches,
// sorted rows and what is small run here.)
//
// A float32 number is the sum of three bfloat16 numbers, x = x1 + x2 + x3 exactly (Henry, Tang, Heinecke, "Leveraging the bfloat16 Artificial
// Intelligence Datatype For Higher-Precision Computations", 2019): x1 is x rounded to nearest, x2 the rest rounded to nearest, |x2| <= 2^-8 |x|,
// x3 what then remains, |x3| <= 2^-17 |x|.  Six of the nine products leave out less than 2^-24 of x·w, of either sign:
//     x1 w1 + (x1 w2 + x2 w1) + (x1 w3 + x2 w2 + x3 w1),
// each exact in the tensor core's fp32 sums.  (Parts that are cut off instead of rounded leave out up to 2^-21, always towards zero.)  The tensor core cuts off when it adds (measured: 6e-8 of a sum of 64 products, 2e-6 of one of
// 2048), so a sum runs over 64 k only, small products first, and the sums of 64 meet in registers in rounded fp32 additions.
// Error against float64 (2-norm, normal operands), FMA kernel -> this one: K 256 2.8e-7 -> 1.3e-7, 1024 5.7e-7 -> 1.4e-7, 2048 8.1e-7 -> 1.6e-7,
// 5464 1.3e-6 -> 1.6e-7.
// An output that comes out infinite or NaN is formed again with FMAs in order of k: an infinite operand has no such parts, and a finite one
// above the largest bfloat16 number rounds to infinity.
//
//   * 8 producer warps read float32 tiles (128 features and BN rows of 64 k), cut them and write the six bfloat16 tiles in the
//     128-byte-swizzled K-major layout; the next tile's loads are in flight meanwhile;
//   * 24 MMAs of 128 x BN x 16 per 64 k (features are the MMA's rows, so that few tokens waste nothing);
//   * 4 epilogue warps, the first of which issues the MMAs, add the finished sum (two in TMEM, alternating) to their registers: a thread
//     owns one feature.
// Few tiles: a cluster of CTAs shares a tile, each takes a part of K; partial sums meet in distributed shared memory in rank order.
// Bound: with many rows the operands' way from the L2 ((128 + BN) x 256 bytes per 128 x BN x 64 products; a kernel that only loads takes
// two thirds of the time) and the six products; with few rows the weights' way from memory.  On one B200, FMA kernel -> this one
// (rows x features x K): 1000 x 6176 x 2048 1060 -> 226 us, 2048 x 1024 x 2048 404 -> 78, 200 x 10928 x 2048 441 -> 141, 200 x 2048 x 5464
// 889 -> 58, 24 x 8192 x 2048 343 -> 29, 12 x 1024 x 4096 370 -> 15, 300 x 1000 x 256 27 -> 13.
#include <cooperative_groups.h>

#include "jllama_b200.h"
#include "linear_f32.cuh"
#include "seq_types.cuh"
#include "tcgen05.cuh"

namespace jl {

constexpr int LF_BM = 128, LF_BK = 64, LF_PROD = 8, LF_THREADS = (LF_PROD + 4) * 32;
constexpr uint32_t LF_A_BYTES = LF_BM * LF_BK * 2;                   // one part of the weights

constexpr uint32_t lf_stage_bytes(int bn) { return 3 * (LF_A_BYTES + bn * LF_BK * 2); }
constexpr int lf_stages(int bn) { return bn <= 32 ? 3 : 2; }
constexpr size_t lf_smem(int bn) { return (size_t)lf_stages(bn) * lf_stage_bytes(bn) + 1024; }

struct LinearF32 {
  const float* x; const float* w; float* out;
  int ldx, ldo, M, N, K, act, splits;
  float p0, p1;
  LinearGroup g;
};

template <int BN>
__global__ void __launch_bounds__(LF_THREADS, 1) linear_f32_kernel(const LinearF32 p) {
  constexpr int STAGES = lf_stages(BN);
  constexpr int STEP = LF_PROD * 4, NW = LF_BM / STEP, NX = BN / STEP;       // rows of the weights and of x per producer thread
  constexpr uint32_t STAGE = lf_stage_bytes(BN), B_BYTES = BN * LF_BK * 2, B_OFF = 3 * LF_A_BYTES;
  constexpr uint32_t COLS = 2 * BN < 32 ? 32 : 2 * BN;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(8) unsigned long long bar_mem[2 * 3 + 4];
  __shared__ uint32_t tmem_slot;
  __shared__ int srow[BN];
  const uint32_t raw = tc::smem_u32(smem_raw), base = (raw + 1023u) & ~1023u, bars = tc::smem_u32(bar_mem);
  auto full = [&](int s) { return bars + 8u * s; };
  auto empty = [&](int s) { return bars + 24 + 8u * s; };
  auto tfull = [&](int s) { return bars + 48 + 8u * s; };
  auto tempty = [&](int s) { return bars + 64 + 8u * s; };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int part = (int)(blockIdx.x % p.splits), n0 = (int)(blockIdx.x / p.splits) * LF_BM, m0 = blockIdx.y * BN;

  if (warp == LF_PROD) {
    tc::tmem_alloc(tc::smem_u32(&tmem_slot), COLS);
    if (lane == 0) {
      for (int s = 0; s < STAGES; ++s) { tc::mbar_init(full(s), LF_PROD); tc::mbar_init(empty(s), 1); }
      for (int s = 0; s < 2; ++s) { tc::mbar_init(tfull(s), 1); tc::mbar_init(tempty(s), 4); }
      tc::fence_barrier_init();
    }
  }
  pdl_wait();
  pdl_launch_dependents();
  const float* x = p.x;
  const float* w = p.w;
  float* out = p.out;
  bool off = false;                                                  // uniform for the cluster: nothing to compute
  if (p.g.tile_group) {
    const int e = p.g.tile_group[m0 / LT_BM];
    off = e < 0;
    w += (long long)(off ? 0 : e) * p.g.w_bs;
  } else {
    const long long z = blockIdx.z;
    const long long e = p.g.w_index ? p.g.w_index[z] : z;
    off = e < 0;
    x += (z / p.g.x_div) * p.g.x_bs;
    w += (off ? 0 : e) * p.g.w_bs;
    out += z * p.g.o_bs;
  }
  for (int i = threadIdx.x; i < BN; i += LF_THREADS) {
    const int gm = m0 + i;
    srow[i] = gm < p.M ? ((p.g.tile_group && p.g.row_src) ? p.g.row_src[gm] : gm) : -1;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const int k_blocks = (p.K + LF_BK - 1) / LF_BK, per = (k_blocks + p.splits - 1) / p.splits;
  const int kb0 = part * per, kb1 = off ? kb0 : min(k_blocks, kb0 + per);

  float* tile = reinterpret_cast<float*>(smem_raw + (base - raw));   // [BN][128], in the ring once it is free
  if (warp < LF_PROD) {
    const int r = threadIdx.x / 8, c = threadIdx.x & 7;              // 8 lanes take the 64 k of a row, 8 each
    // rows beyond the matrix repeat another one: their outputs are not stored (padding rows: stored as zero)
    const float* src[NW + NX];
#pragma unroll
    for (int i = 0; i < NW; ++i) src[i] = w + (size_t)min(n0 + r + i * STEP, p.N - 1) * p.K + 8 * c;
#pragma unroll
    for (int i = 0; i < NX; ++i) src[NW + i] = x + (size_t)max(srow[r + i * STEP], 0) * p.ldx + 8 * c;
    float4 va[NW + NX], vb[NW + NX];                                 // the next block of 64 k
    auto load = [&](int kb) {
      if (kb >= kb1) return;
      const size_t at = (size_t)kb * LF_BK;
      if ((kb + 1) * LF_BK <= p.K) {
#pragma unroll
        for (int i = 0; i < NW + NX; ++i) {
          va[i] = *reinterpret_cast<const float4*>(src[i] + at);
          vb[i] = *reinterpret_cast<const float4*>(src[i] + at + 4);
        }
      } else {                                                       // the last block: K is a multiple of four
        const bool ina = (int)at + 8 * c < p.K, inb = (int)at + 8 * c + 4 < p.K;
#pragma unroll
        for (int i = 0; i < NW + NX; ++i) {
          va[i] = ina ? *reinterpret_cast<const float4*>(src[i] + at) : make_float4(0.f, 0.f, 0.f, 0.f);
          vb[i] = inb ? *reinterpret_cast<const float4*>(src[i] + at + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
    };
    int stage = 0;
    uint32_t ph = 1;
    const uint32_t lane_off = base + r * 128 + ((c ^ (r & 7)) << 4);         // (STEP rows further: the same swizzle)
    auto put = [&] {
      tc::mbar_wait(empty(stage), ph);
      const uint32_t st = lane_off + stage * STAGE;
#pragma unroll
      for (int i = 0; i < NW + NX; ++i) {
        uint4 h[3];
        lf_split8(va[i], vb[i], h);
        const uint32_t dst = st + (i < NW ? i * STEP * 128 : B_OFF + (i - NW) * STEP * 128);
#pragma unroll
        for (int k = 0; k < 3; ++k)
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + k * (i < NW ? LF_A_BYTES : B_BYTES)), "r"(h[k].x), "r"(h[k].y),
                       "r"(h[k].z), "r"(h[k].w) : "memory");
      }
    };
    auto publish = [&] {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // these writes -> visible to the tensor core
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(full(stage));
      if (++stage == STAGES) { stage = 0; ph ^= 1; }
    };
    load(kb0);
    for (int kb = kb0; kb < kb1; ++kb) {
      put();
      load(kb + 1);
      publish();
    }
  } else {
    // the first epilogue warp also issues: the MMAs of the next 64 k go out before it waits for the current sum
    constexpr uint32_t IDESC = tc::idesc_bf16_f32(LF_BM, BN);
    auto issue = [&](int kb) {
      const int it = kb - kb0, buf = it & 1, stage = it % STAGES;
      tc::mbar_wait(tempty(buf), ((it >> 1) & 1) ^ 1);
      tc::mbar_wait(full(stage), (it / STAGES) & 1);
      tc::fence_after_sync();
      if (tc::elect_one()) {
        const uint32_t sa = base + stage * STAGE, sb = sa + B_OFF;
        const uint32_t d = tmem + buf * BN;
        // parts of the weights and of the rows, the smallest products first
        constexpr int PA[6] = {0, 2, 1, 0, 1, 0}, PB[6] = {2, 0, 1, 1, 0, 0};
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          const uint64_t da = tc::smem_desc_kmajor_sw128(sa + PA[q] * LF_A_BYTES), db = tc::smem_desc_kmajor_sw128(sb + PB[q] * B_BYTES);
#pragma unroll
          for (int k = 0; k < LF_BK / 16; ++k) tc::mma_ss(d, da + 2 * k, db + 2 * k, IDESC, q != 0 || k != 0);
        }
        tc::mma_commit(empty(stage));
        tc::mma_commit(tfull(buf));
      }
      __syncwarp();
    };
    const uint32_t row = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    float acc[BN];                                                   // one feature, BN rows
#pragma unroll
    for (int j = 0; j < BN; ++j) acc[j] = 0.0f;
    if (warp == LF_PROD && kb0 < kb1) issue(kb0);
    for (int kb = kb0; kb < kb1; ++kb) {
      const int it = kb - kb0, buf = it & 1;
      if (warp == LF_PROD && kb + 1 < kb1) issue(kb + 1);
      tc::mbar_wait(tfull(buf), (it >> 1) & 1);
      tc::fence_after_sync();
#pragma unroll
      for (int c0 = 0; c0 < BN; c0 += 16) {
        uint32_t v[16];
        tc::tmem_ld16(row + buf * BN + c0, v);
        tc::tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[c0 + j] += __uint_as_float(v[j]);
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(tempty(buf));
    }
    // every MMA has completed (the last sum is here): the ring takes the tile
#pragma unroll
    for (int j = 0; j < BN; ++j) tile[j * LF_BM + (warp & 3) * 32 + lane] = acc[j];
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == LF_PROD) tc::tmem_dealloc(tmem, COLS);
  if (off) return;

  // an output that is not finite: the same sum with FMAs in order of k
  auto finish = [&](float s, int m, int n) {
    const int r = srow[m];
    if (r < 0) {
      s = 0.0f;
    } else if (!(fabsf(s) < INFINITY)) {
      const float* xr = x + (size_t)r * p.ldx;
      const float* wr = w + (size_t)n * p.K;
      s = 0.0f;
      for (int k = 0; k < p.K; ++k) s = fmaf(xr[k], wr[k], s);
    }
    return apply_act(s, p.act, p.p0, p.p1);
  };
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  if (p.splits > 1) cl.sync();
  const int rows = (BN + p.splits - 1) / p.splits, r1 = min(BN, (part + 1) * rows);
  for (int i = part * rows * LF_BM + threadIdx.x; i < r1 * LF_BM; i += LF_THREADS) {
    const int j = i / LF_BM, n = n0 + i % LF_BM;
    if (m0 + j >= p.M || n >= p.N) continue;
    float s = 0.0f;
    if (p.splits == 1) s = tile[i];
    else for (int q = 0; q < p.splits; ++q) s += cl.map_shared_rank(tile, q)[i];
    out[(size_t)(m0 + j) * p.ldo + n] = finish(s, j, n);
  }
  if (p.splits > 1) cl.sync();                                       // no CTA leaves while its tile may still be read
}

template <int BN>
static cudaError_t lf_launch(const LinearF32& p, int nbatch, cudaStream_t st) {
  auto* kernel = linear_f32_kernel<BN>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lf_smem(BN));
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((p.N + LF_BM - 1) / LF_BM * p.splits), (unsigned)((p.M + BN - 1) / BN), p.g.tile_group ? 1u : (unsigned)nbatch);
  cfg.blockDim = dim3(LF_THREADS);
  cfg.dynamicSmemBytes = lf_smem(BN);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (p.splits > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = p.splits;
    attr[na].val.clusterDim.y = 1;
    attr[na++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kernel, p);
}

// From 9 rows (up to 8 the weight-streaming kernel reads the weights once at the rate of memory) and from K 256 on (four sums of 64: below,
// the FMA kernel's error is as small); 16-byte loads along K.
bool linear_f32_takes(int M, int K, int ldx, const LinearGroup& g, const void* x, const void* w) {
  return M > 8 && K >= 256 && K % 4 == 0 && ldx % 4 == 0 && g.x_bs % 4 == 0 && g.w_bs % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
}

// Rows per tile and parts of K: the least time of the busiest SM in cycles, from what a CTA takes per 64 k, to begin and end, and to
// meet its cluster (fitted to the times above and their neighbours; clusters of eight wait for a place).
static LinearF32Plan lf_plan(int M, int N, int K, int nbatch, bool sorted) {
  static const struct { int bn; double cycles; } shapes[] = {{32, 2000.0}, {64, 2300.0}, {128, 3400.0}};
  const int k_blocks = (K + LF_BK - 1) / LF_BK;
  double best = 1e300;
  LinearF32Plan p{64, 1, 0, 0};
  for (const auto& sh : shapes) {
    const long tiles = (long)((M + sh.bn - 1) / sh.bn) * ((N + LF_BM - 1) / LF_BM) * nbatch;
    if (sorted && sh.bn > LT_BM) continue;
    for (int s = 1; s <= 8; s *= 2) {
      if (s > 1 && k_blocks / s < 2) break;
      const double t = (double)((tiles * s + SMS - 1) / SMS) * (4000.0 + sh.cycles * ((k_blocks + s - 1) / s) + (s == 1 ? 0.0 : s < 8 ? 5000.0 : 9000.0));
      if (t < best) { best = t; p = {sh.bn, s, (k_blocks + s - 1) / s, tiles}; }
    }
  }
  return p;
}

LinearF32Plan linear_f32_plan(int M, int N, int K) { return lf_plan(M, N, K, 1, false); }

cudaError_t linear_f32_launch(const float* x, int ldx, const float* w, float* out, int ldo, int M, int N, int K, int act, float p0, float p1,
                              cudaStream_t st, const LinearGroup& g, int nbatch) {
  const LinearF32Plan plan = lf_plan(M, N, K, g.tile_group ? 1 : nbatch, g.tile_group != nullptr);
  const LinearF32 p{x, w, out, ldx, ldo, M, N, K, act, plan.splits, p0, p1, g};
  if (plan.bn == 32) return lf_launch<32>(p, nbatch, st);
  if (plan.bn == 64) return lf_launch<64>(p, nbatch, st);
  return lf_launch<128>(p, nbatch, st);
}

}  // namespace jl

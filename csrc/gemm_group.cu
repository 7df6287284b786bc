// bf16 GEMM on tcgen05 over sorted rows, with what follows it in the epilogue: a mixture of experts over a prompt, and gated layers.
//
// x [M, K]: every 128-row tile belongs to one of `groups` weight matrices (tile_group; none: one matrix).  Forms of the result:
//   GG_F32   fp32 [M, N]
//   GG_BF16  bf16 [M, N], an activation on the rounded value
//   GG_GLU   bf16 [M, F]: glu(gate_j, up_j) of two parts of the weight matrix, F rows from g_off and F rows from u_off.  A tile's 256 weight rows
//            are 128 of each, so a thread holds both halves of its 128 results: the fp32 gate | up product never goes to memory.
// One persistent CTA per SM: tiles of 128 x 256, A-tile index fastest (tiles that run together share weights through L2), TMA ring of four 64-k stages,
// one MMA thread, accumulators double-buffered over all 512 TMEM columns, eight epilogue warps; results leave through shared memory as TMA stores of whole
// 128-byte rows (16 bytes a lane straight from registers, a row per lane, cost the fp32 form half its time).
// Exact float32 activations (this file is compiled without fast math).
// Bound: the operands' way from L2 (48 KB per 512 cycles of products) and, for few k, the activations of eight warps.  One B200, gate | up product (fp32) and
// activation pass -> one kernel (tokens x F x K): 2048 x 5464 x 2048 94 -> 68 us (1340 TFLOP/s), 2048 x 1360 x 2048 34 -> 26.5, 512 x 2736 x 2048 20 -> 16, 129 x 1024 x 1024
// 13.7 -> 10.5, the same bits; 2048 tokens x top 4 of 32 experts of 2048 x 1024 with a shared one: both GEMMs and activations 265 -> 190 us, the layer 337 -> 275 between events.
#include "jllama_b200.h"
#include "seq_types.cuh"
#include "tcgen05.cuh"

namespace jl {

constexpr int GG_BM = 128, GG_BN = 256, GG_BK = 64, GG_THREADS = 384, GG_STAGES = 4;        // warps: 0 TMA, 1 MMA, 2 TMEM, 4-11 epilogue
constexpr uint32_t GG_A_BYTES = GG_BM * GG_BK * 2, GG_B_BYTES = GG_BN * GG_BK * 2, GG_STAGE = GG_A_BYTES + GG_B_BYTES;
constexpr uint32_t GG_EPI = 8 * 4096;                          // eight warps x 32 rows x 128 bytes
constexpr size_t GG_SMEM = GG_STAGES * GG_STAGE + GG_EPI + 8 * (2 * GG_STAGES + 4) + 16 + 1024;

enum { GG_F32 = 0, GG_BF16 = 1, GG_GLU = 2 };
constexpr int GG_CLAMPED = -1, GG_ANY = -2;                      // activations beside ACT_*: the clamped form (GG_GLU), one named at run time

struct GroupGemm {
  int K, N, a_blocks, b_blocks;      // N: columns of the result
  int g_off, u_off, group_rows;      // GG_GLU: first gate and up row; weight rows per matrix
  const int* tile_group;             // matrix of an A tile (< 0: padding, any will do), or nullptr
  const int* a_blocks_used;          // optional device count of leading A tiles that hold rows
  int kind, act;
  float limit, alpha;
  void* narrow;                      // result of fewer than 32 columns off the 16-byte boundary (GG_F32, GG_BF16): stored element by element; else nullptr
};

template <int ACT>
__device__ __forceinline__ float gg_act(float z, const GroupGemm& p) { return apply_act(z, ACT == GG_ANY ? p.act : ACT, 0.0f, 0.0f); }
template <int ACT>
__device__ __forceinline__ float gg_glu(float g, float u, const GroupGemm& p) {
  if constexpr (ACT != GG_CLAMPED) return gg_act<ACT>(g, p) * u;
  g = fminf(g, p.limit);
  u = fminf(fmaxf(u, -p.limit), p.limit);
  return g * sigmoid_f(p.alpha * g) * (u + 1.0f);
}
__device__ __forceinline__ void gg_store(const CUtensorMap* map, uint32_t src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(c0),
               "r"(c1) : "memory");
}

// ACT: the activation, known at compile time: a switch per value leaves nothing to overlap (whole launches, gated relu
// 59.7 -> 25.1 us for 2048 x 1360 x 2048 and 152 -> 71 for F 5464; product and activation pass 31.9 and 97).  Only the two activations that take numbers of their
// own, which no layer puts here, are named at run time (GG_ANY).
template <int EPI, int ACT>
__global__ void __launch_bounds__(GG_THREADS, 1)
gemm_group_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                  const __grid_constant__ CUtensorMap tmap_out, const GroupGemm p) {
  extern __shared__ uint8_t smem_raw[];
  constexpr uint32_t IDESC = tc::idesc_bf16_f32(GG_BM, GG_BN);
  constexpr int OUT_COLS = EPI == GG_GLU ? GG_BN / 2 : GG_BN;    // columns of the result that a tile gives
  const uint32_t base = (tc::smem_u32(smem_raw) + 1023u) & ~1023u, epi = base + GG_STAGES * GG_STAGE, bars = epi + GG_EPI;
  auto full = [&](int s) { return bars + 8u * s; };
  auto empty = [&](int s) { return bars + 8u * (GG_STAGES + s); };
  auto tfull = [&](int s) { return bars + 8u * (2 * GG_STAGES + s); };
  auto tempty = [&](int s) { return bars + 8u * (2 * GG_STAGES + 2 + s); };
  const uint32_t tmem_slot = bars + 8u * (2 * GG_STAGES + 4);
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - tc::smem_u32(smem_raw)));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_kb = (p.K + GG_BK - 1) / GG_BK;

  if (warp == 0 && lane == 0) { tc::prefetch_tensormap(&tmap_a); tc::prefetch_tensormap(&tmap_b); tc::prefetch_tensormap(&tmap_out); }
  if (warp == 1 && lane == 0) {
    for (int s = 0; s < GG_STAGES; ++s) { tc::mbar_init(full(s), 1); tc::mbar_init(empty(s), 1); }
    for (int s = 0; s < 2; ++s) { tc::mbar_init(tfull(s), 1); tc::mbar_init(tempty(s), 8); }
    tc::fence_barrier_init();
  }
  if (warp == 2) tc::tmem_alloc(tmem_slot, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot_ptr;
  pdl_wait();                                               // everything above overlapped the previous kernel's tail
  pdl_launch_dependents();
  int a_blocks = p.a_blocks;
  if (p.a_blocks_used != nullptr) {                         // one value for every thread of the grid: all roles walk the same list
    const int used = *p.a_blocks_used;
    a_blocks = used < 1 ? 1 : (used < a_blocks ? used : a_blocks);
  }
  const int num_tiles = a_blocks * p.b_blocks;

  if (warp == 0) {
    // ===================================================== TMA producer
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
        const int b_blk = t / a_blocks, a_blk = t % a_blocks;
        int row = 0;
        if (p.tile_group != nullptr) {
          const int e = p.tile_group[a_blk];
          row = (e < 0 ? 0 : e) * p.group_rows;
        }
        const int r0 = row + (EPI == GG_GLU ? p.g_off + b_blk * (GG_BN / 2) : b_blk * GG_BN);
        const int r1 = EPI == GG_GLU ? row + p.u_off + b_blk * (GG_BN / 2) : r0 + GG_BN / 2;
        for (int kb = 0; kb < num_kb; ++kb) {
          const uint32_t sa = base + stage * GG_STAGE, sb = sa + GG_A_BYTES;
          tc::mbar_wait(empty(stage), phase ^ 1);
          tc::mbar_expect_tx(full(stage), GG_STAGE);
          tc::tma_load_2d(sa, &tmap_a, full(stage), kb * GG_BK, a_blk * GG_BM, tc::EVICT_NORMAL);
          tc::tma_load_2d(sb, &tmap_b, full(stage), kb * GG_BK, r0, tc::EVICT_LAST);
          tc::tma_load_2d(sb + GG_B_BYTES / 2, &tmap_b, full(stage), kb * GG_BK, r1, tc::EVICT_LAST);
          if (++stage == GG_STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ===================================================== MMA issuer (single thread)
    if (lane == 0) {
      int stage = 0, it = 0; uint32_t phase = 0;
      for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it) {
        const int as = it & 1;
        tc::mbar_wait(tempty(as), ((it >> 1) & 1) ^ 1);     // the epilogue has drained this accumulator
        tc::fence_after_sync();
        const uint32_t d = tmem + as * GG_BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          tc::mbar_wait(full(stage), phase);
          tc::fence_after_sync();
          const uint32_t sa = base + stage * GG_STAGE;
          const uint64_t da = tc::smem_desc_kmajor_sw128(sa), db = tc::smem_desc_kmajor_sw128(sa + GG_A_BYTES);
#pragma unroll
          for (int k = 0; k < GG_BK / 16; ++k) tc::mma_ss(d, da + 2 * k, db + 2 * k, IDESC, kb != 0 || k != 0);
          tc::mma_commit(empty(stage));
          if (++stage == GG_STAGES) { stage = 0; phase ^= 1; }
        }
        tc::mma_commit(tfull(as));
      }
    }
  } else if (warp >= 4) {
    // ===================================================== epilogue: a token row per thread; TMEM -> registers -> shared -> TMA store
    const int quarter = warp & 3, part = (warp >> 2) - 1;    // rows 32 quarter ..; half of the tile's columns
    const uint32_t mine = epi + (warp - 4) * 4096;
    uint8_t* my_ptr = smem_raw + (mine - tc::smem_u32(smem_raw));
    int it = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it) {
      const int b_blk = t / a_blocks, a_blk = t % a_blocks, as = it & 1, row0 = a_blk * GG_BM + quarter * 32, col0 = b_blk * OUT_COLS;
      tc::mbar_wait(tfull(as), (it >> 1) & 1);
      tc::fence_after_sync();
      const uint32_t t_row = tmem + ((uint32_t)(quarter * 32) << 16) + as * GG_BN;
      constexpr int STEP = EPI == GG_F32 ? 32 : 64;         // columns of a 128-byte row
#pragma unroll 1
      for (int c0 = part * (OUT_COLS / 2); c0 < (part + 1) * (OUT_COLS / 2); c0 += STEP) {
        uint4 w[8];
#pragma unroll
        for (int h = 0; h < STEP / 32; ++h) {
          uint32_t v[32];
          tc::tmem_ld32(t_row + c0 + h * 32, v);
          if constexpr (EPI == GG_GLU) {
            uint32_t u[32];
            tc::tmem_ld32(t_row + GG_BN / 2 + c0 + h * 32, u);
            tc::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint32_t r[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int e = 8 * j + 2 * i;
                r[i] = pack_bf16(gg_glu<ACT>(__uint_as_float(v[e]), __uint_as_float(u[e]), p), gg_glu<ACT>(__uint_as_float(v[e + 1]), __uint_as_float(u[e + 1]), p));
              }
              w[h * 4 + j] = make_uint4(r[0], r[1], r[2], r[3]);
            }
          } else if constexpr (EPI == GG_BF16) {
            tc::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint32_t r[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                r[i] = pack_bf16(__uint_as_float(v[8 * j + 2 * i]), __uint_as_float(v[8 * j + 2 * i + 1]));
                if constexpr (ACT != ACT_NONE) r[i] = pack_bf16(gg_act<ACT>(bf16_lo(r[i]), p), gg_act<ACT>(bf16_hi(r[i]), p));
              }
              w[h * 4 + j] = make_uint4(r[0], r[1], r[2], r[3]);
            }
          } else {
            tc::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 8; ++j) w[j] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          }
        }
        if constexpr (EPI != GG_GLU) {
          if (p.narrow != nullptr) {
            constexpr int ES = EPI == GG_F32 ? 4 : 2;
            const uint32_t* e = reinterpret_cast<const uint32_t*>(w);
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (col0 + c0 + j < p.N) {
                uint8_t* o = reinterpret_cast<uint8_t*>(p.narrow) + ((size_t)(row0 + lane) * p.N + col0 + c0 + j) * ES;
                if constexpr (EPI == GG_F32) *reinterpret_cast<uint32_t*>(o) = e[j];
                else *reinterpret_cast<unsigned short*>(o) = (unsigned short)(e[j / 2] >> (16 * (j & 1)));
              }
            continue;
          }
        }
        // the store before must have finished reading the buffer
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
        uint8_t* dst = my_ptr + lane * 128;
#pragma unroll
        for (int j = 0; j < 8; ++j) *reinterpret_cast<uint4*>(dst + ((j ^ (lane & 7)) << 4)) = w[j];      // 16-byte chunks, swizzled as the map expects
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          // rows and columns beyond the result are clipped; a box that lies beyond the last column is not sent at all
          if (col0 + c0 < p.N) gg_store(&tmap_out, mine, col0 + c0, row0);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(tempty(as));
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");        // stores complete before exit
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 2) tc::tmem_dealloc(tmem, 512);
}

using GroupKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const GroupGemm);
template <int EPI>
static GroupKernel group_kernel(int act) {
  switch (act) {
    case ACT_NONE: return gemm_group_kernel<EPI, ACT_NONE>;
    case ACT_RELU2: return gemm_group_kernel<EPI, ACT_RELU2>;
    case ACT_GELU_TANH: return gemm_group_kernel<EPI, ACT_GELU_TANH>;
    case ACT_SILU: return gemm_group_kernel<EPI, ACT_SILU>;
    case ACT_SIGMOID: return gemm_group_kernel<EPI, ACT_SIGMOID>;
    case ACT_RELU: return gemm_group_kernel<EPI, ACT_RELU>;
    default: return gemm_group_kernel<EPI, GG_ANY>;
  }
}

static int group_launch(int epi, const void* x, const void* w, void* out, int M, GroupGemm p, int w_rows, int num_sms, cudaStream_t st) {
  CUtensorMap ta, tb, to;
  int rc;
  if ((rc = make_tmap_2d_bf16(&ta, x, M, p.K, p.K, GG_BM))) return rc;
  if ((rc = make_tmap_2d_bf16(&tb, w, w_rows, p.K, p.K, GG_BN / 2))) return rc;
  if (epi != GG_GLU && p.N < 32 && ((uintptr_t)out & 15) != 0) {
    JL_CHECK_ARG((uintptr_t)out % (epi == GG_F32 ? 4 : 2) == 0, "jl_gemm_grouped: result off its elements' boundary");
    p.narrow = out;
    to = tb;                                                 // (not used)
  } else if ((rc = epi == GG_F32 ? make_tmap_2d_f32(&to, out, M, p.N, p.N, 32) : make_tmap_2d_bf16(&to, out, M, p.N, p.N, 32))) {
    return rc;
  }
  const int cols = epi == GG_GLU ? GG_BN / 2 : GG_BN;
  p.a_blocks = (M + GG_BM - 1) / GG_BM;
  p.b_blocks = (p.N + cols - 1) / cols;
  const long tiles = (long)p.a_blocks * p.b_blocks;
  auto* kern = epi == GG_F32 ? gemm_group_kernel<GG_F32, ACT_NONE> : epi == GG_BF16 ? group_kernel<GG_BF16>(p.act)
               : p.kind == 1 ? gemm_group_kernel<GG_GLU, GG_CLAMPED> : group_kernel<GG_GLU>(p.act);
  JL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GG_SMEM));
  JL_CUDA(launch_pdl(kern, dim3((unsigned)(tiles < num_sms ? tiles : num_sms)), dim3(GG_THREADS), GG_SMEM, st, ta, tb, to, p));
  return JL_OK;
}

}  // namespace jl

using namespace jl;

// x [M, K] with M a multiple of 128 and every 128-row tile belonging to one of `groups` weight matrices w [groups][N, K]; out[m] =
// act(W_(tile_group[m / 128]) x[m]) (fp32, no activation; or bf16, the activation on the rounded value; row pitch N).  tiles_used (optional, device): how
// many leading 128-row tiles hold rows; the rest are not computed.
static int grouped(const void* x, const void* w, void* out, int M, int N, int K, int groups, const int* tile_group, const int* tiles_used, int out_f32,
                   int act, int num_sms, void* stream) {
  JL_CHECK_ARG(M >= GG_BM && M % GG_BM == 0, "jl_gemm_grouped: M=%d must be a multiple of %d", M, GG_BM);
  JL_CHECK_ARG(N >= 8 && N % 8 == 0 && K >= 8 && K % 8 == 0 && groups >= 1 && tile_group != nullptr,
               "jl_gemm_grouped: bad shape N=%d K=%d groups=%d", N, K, groups);
  JL_CHECK_ARG(act >= 0 && act <= ACT_LAST && (act == ACT_NONE || !out_f32), "jl_gemm_grouped: bad activation %d", act);
  GroupGemm p{};
  p.K = K; p.N = N; p.group_rows = N;
  p.tile_group = tile_group; p.a_blocks_used = tiles_used; p.act = act;
  return group_launch(out_f32 ? GG_F32 : GG_BF16, x, w, out, M, p, N * groups, num_sms > 0 ? num_sms : 148, (cudaStream_t)stream);
}
extern "C" JL_API int jl_gemm_grouped(const void* x, const void* w, void* out, int M, int N, int K, int groups, const int* tile_group,
                                      const int* tiles_used, int out_f32, int num_sms, void* stream) {
  return grouped(x, w, out, M, N, K, groups, tile_group, tiles_used, out_f32, ACT_NONE, num_sms, stream);
}
extern "C" JL_API int jl_gemm_grouped_act(const void* x, const void* w, void* out, int M, int N, int K, int groups, const int* tile_group,
                                          const int* tiles_used, int act, int num_sms, void* stream) {
  return grouped(x, w, out, M, N, K, groups, tile_group, tiles_used, 0, act, num_sms, stream);
}

// out [M, F] (bf16) = glu(gate, up): the fp32 products of x [M, K] with F weight rows from g_off and F from u_off of w [groups][w_rows, K]; kind and what goes
// with it as in jl_glu_act.  tile_group nullptr: one matrix, any M.
extern "C" JL_API int jl_gemm_glu(const void* x, const void* w, void* out, int M, int F, int K, int w_rows, int g_off, int u_off, int groups,
                                  const int* tile_group, const int* tiles_used, int kind, int act, float limit, float alpha, int num_sms, void* stream) {
  JL_CHECK_ARG(M >= 1 && F >= 8 && F % 8 == 0 && K >= 8 && K % 8 == 0 && groups >= 1, "jl_gemm_glu: bad shape M=%d F=%d K=%d", M, F, K);
  JL_CHECK_ARG(g_off >= 0 && u_off >= 0 && g_off + F <= w_rows && u_off + F <= w_rows, "jl_gemm_glu: rows %d and %d of %d", g_off, u_off, w_rows);
  JL_CHECK_ARG(tile_group == nullptr ? groups == 1 : M % GG_BM == 0, "jl_gemm_glu: sorted rows come in tiles of %d, M=%d", GG_BM, M);
  JL_CHECK_ARG(kind == 0 || kind == 1, "jl_gemm_glu: bad kind %d", kind);
  JL_CHECK_ARG(act >= 0 && act <= ACT_LAST, "jl_gemm_glu: bad activation %d", act);
  GroupGemm p{};
  p.K = K; p.N = F; p.group_rows = w_rows; p.g_off = g_off; p.u_off = u_off;
  p.tile_group = tile_group; p.a_blocks_used = tiles_used;
  p.kind = kind; p.act = act; p.limit = limit; p.alpha = alpha;
  return group_launch(GG_GLU, x, w, out, M, p, w_rows * groups, num_sms > 0 ? num_sms : 148, (cudaStream_t)stream);
}

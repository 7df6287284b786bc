// bf16 GEMM on 5th-generation tensor cores: D = A[Ra,K] · B[Rb,K]^T with fp32 accumulation in TMEM.
//
//   * operands are K-major and arrive by TMA (128-byte swizzle) into a multi-stage mbarrier ring;
//   * one elected thread issues tcgen05.mma (UMMA 128 x BN x 16), completion is signalled with
//     tcgen05.commit → mbarrier, the accumulator (double-buffered, 2·BN TMEM columns) is drained by four
//     epilogue warps with tcgen05.ld while the next tile's MMAs run;
//   * persistent: one CTA per SM walks the tile list, A-tile index fastest so CTAs that run together
//     share the same weight tile through L2.
//
// A = activations [M,K], B = weights [N,K]; D tile rows are tokens (prefill).  With few tokens the weights take the MMA's rows
// instead (gemm_swap.cu).
// Epilogues: plain bf16 / fp32, residual add, SwiGLU over interleaved (w1,w3) output columns.
//
// Replaces the cuBLAS GEMMs XLA emitted for jax_llama/model.py:119-150 (wq/wk/wv/wo),
// :311-338 (w1/w2/w3) and :699-706 (lm_head).
#include <stdlib.h>

#include "gemm_swap.cuh"
#include "jllama_b200.h"
#include "tcgen05.cuh"

namespace jl {

int gemm_2cta_f32(const void* x, const void* w, void* out, int M, int N, int K, int num_sms, void* stream);      // gemm_2cta.cu

constexpr int GEMM_BM = 128;
constexpr int GEMM_BK = 64;
constexpr int GEMM_THREADS = 256;   // warp0 TMA, warp1 MMA, warp2 TMEM alloc, warp3 idle, warps 4-7 epilogue

enum { EPI_PLAIN = 0, EPI_RESIDUAL = 1, EPI_SWIGLU = 2 };

struct GemmParams {
  void* out;
  const __nv_bfloat16* residual;
  int Ra, Rb, K;            // A-side rows, B-side rows, reduction length
  int ldo;                  // output row pitch (elements)
  int a_blocks, b_blocks;   // tile counts
  int stages;
  uint64_t hint_a, hint_b;
  unsigned long long* trace;         // optional [grid][16] %globaltimer stamps (jl_gemm_set_trace), NULL = off
};

// one thread records when it reached a point of the kernel (scripts/gemm_trace.py prints the timeline)
__device__ __forceinline__ void gemm_stamp(const GemmParams& p, int ev) {
  if (p.trace != nullptr) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    p.trace[(size_t)blockIdx.x * 16 + ev] = t;
  }
}

template <int BN, int EPI, bool OUT_F32>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  constexpr uint32_t A_BYTES = GEMM_BM * GEMM_BK * 2;
  constexpr uint32_t B_BYTES = BN * GEMM_BK * 2;
  constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr uint32_t TMEM_COLS = 2 * BN;                    // 256 or 512, double-buffered
  constexpr uint32_t IDESC = tc::idesc_bf16_f32(GEMM_BM, BN);

  const uint32_t smem_base = (tc::smem_u32(smem_raw) + 1023u) & ~1023u;
  const int stages = p.stages;
  const uint32_t bars = smem_base + stages * STAGE_BYTES;       // full[stages] | empty[stages] | tfull[2] | tempty[2]
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (stages + s); };
  auto tfull_bar = [&](int s) { return bars + 8u * (2 * stages + s); };
  auto tempty_bar = [&](int s) { return bars + 8u * (2 * stages + 2 + s); };
  const uint32_t tmem_slot = bars + 8u * (2 * stages + 4);
  volatile uint32_t* tmem_slot_ptr =
      reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - tc::smem_u32(smem_raw)));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_kb = (p.K + GEMM_BK - 1) / GEMM_BK;

  if (threadIdx.x == 0) gemm_stamp(p, 0);
  if (warp == 0 && lane == 0) {
    tc::prefetch_tensormap(&tmap_a);
    tc::prefetch_tensormap(&tmap_b);
  }
  if (warp == 1 && lane == 0) {
    for (int s = 0; s < stages; ++s) { tc::mbar_init(full_bar(s), 1); tc::mbar_init(empty_bar(s), 1); }
    for (int s = 0; s < 2; ++s) { tc::mbar_init(tfull_bar(s), 1); tc::mbar_init(tempty_bar(s), 4); }
    tc::fence_barrier_init();
  }
  if (warp == 2) tc::tmem_alloc(tmem_slot, TMEM_COLS);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = *tmem_slot_ptr;
  if (threadIdx.x == 0) gemm_stamp(p, 1);

  pdl_wait();                 // everything above overlapped the previous kernel's tail
  pdl_launch_dependents();
  const int a_blocks = p.a_blocks;
  const int num_tiles = a_blocks * p.b_blocks;

  if (warp == 0) {
    // ===================================================== TMA producer
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      gemm_stamp(p, 2);
      for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
        const int b_blk = t / a_blocks;
        const int a_blk = t % a_blocks;
        const int b_row = b_blk * BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          const uint32_t sa = smem_base + stage * STAGE_BYTES, sb = sa + A_BYTES;
          tc::mbar_wait(empty_bar(stage), phase ^ 1);
          tc::mbar_expect_tx(full_bar(stage), A_BYTES + B_BYTES);
          tc::tma_load_2d(sa, &tmap_a, full_bar(stage), kb * GEMM_BK, a_blk * GEMM_BM, p.hint_a);
          tc::tma_load_2d(sb, &tmap_b, full_bar(stage), kb * GEMM_BK, b_row, p.hint_b);
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ===================================================== MMA issuer (single thread)
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0; int it = 0;
      for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it) {
        const int as = it & 1; const uint32_t aphase = (it >> 1) & 1;
        tc::mbar_wait(tempty_bar(as), aphase ^ 1);          // epilogue has drained this accumulator
        tc::fence_after_sync();
        const uint32_t d_tmem = tmem_base + as * BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          tc::mbar_wait(full_bar(stage), phase);
          tc::fence_after_sync();
          if (it == 0 && kb == 0) gemm_stamp(p, 3);
          const uint32_t sa = smem_base + stage * STAGE_BYTES, sb = sa + A_BYTES;
          const uint64_t da = tc::smem_desc_kmajor_sw128(sa), db = tc::smem_desc_kmajor_sw128(sb);
#pragma unroll
          for (int k = 0; k < GEMM_BK / 16; ++k)            // +32 bytes per UMMA_K inside the swizzle span
            tc::mma_ss(d_tmem, da + 2 * k, db + 2 * k, IDESC, kb != 0 || k != 0);
          tc::mma_commit(empty_bar(stage));                 // frees the smem slot when these MMAs retire
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
        tc::mma_commit(tfull_bar(as));                      // accumulator complete → epilogue
        if (it == 0) gemm_stamp(p, 4);
      }
    }
  } else if (warp >= 4) {
    // ===================================================== epilogue: TMEM → registers → global
    const int quarter = warp & 3;                           // TMEM lanes [32·quarter, 32·quarter+32)
    int it = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it) {
      const int b_blk = t / a_blocks;
      const int a_blk = t % a_blocks;
      const int as = it & 1; const uint32_t aphase = (it >> 1) & 1;
      tc::mbar_wait(tfull_bar(as), aphase);
      tc::fence_after_sync();
      if (it == 0 && threadIdx.x == 128) gemm_stamp(p, 5);
      const int ra = a_blk * GEMM_BM + quarter * 32 + lane;  // A-side row of this thread
      const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + as * BN;
      constexpr int CH = 32;
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += CH) {
        uint32_t v[CH];
        tc::tmem_ld32(t_row + c0, v);
        tc::tmem_ld_wait();
        const int cb0 = b_blk * BN + c0;                    // first B-side row of this chunk
        // thread owns one token row, CH consecutive output columns
        if (ra < p.Ra) {
          if constexpr (EPI == EPI_SWIGLU) {
            __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)ra * p.ldo + cb0 / 2;
            uint32_t w[CH / 4];
#pragma unroll
            for (int j = 0; j < CH / 4; ++j) {
              float g0 = __bfloat162float(__float2bfloat16(__uint_as_float(v[4 * j])));
              float u0 = __bfloat162float(__float2bfloat16(__uint_as_float(v[4 * j + 1])));
              float g1 = __bfloat162float(__float2bfloat16(__uint_as_float(v[4 * j + 2])));
              float u1 = __bfloat162float(__float2bfloat16(__uint_as_float(v[4 * j + 3])));
              w[j] = pack_bf16(silu(g0) * u0, silu(g1) * u1);
            }
            if (cb0 + CH <= p.Rb) {
#pragma unroll
              for (int j = 0; j < CH / 16; ++j)
                reinterpret_cast<uint4*>(o)[j] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
            } else {
              for (int j = 0; j < CH / 2; ++j)
                if (cb0 + 2 * j + 1 < p.Rb)
                  o[j] = reinterpret_cast<__nv_bfloat16*>(w)[j];
            }
          } else if constexpr (OUT_F32) {
            float* o = reinterpret_cast<float*>(p.out) + (size_t)ra * p.ldo + cb0;
            if (cb0 + CH <= p.Rb) {
#pragma unroll
              for (int j = 0; j < CH / 4; ++j)
                reinterpret_cast<uint4*>(o)[j] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            } else {
              for (int j = 0; j < CH; ++j) if (cb0 + j < p.Rb) o[j] = __uint_as_float(v[j]);
            }
          } else {
            __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)ra * p.ldo + cb0;
            const bool full = cb0 + CH <= p.Rb;
            uint32_t w[CH / 2];
            if constexpr (EPI == EPI_RESIDUAL) {
              const __nv_bfloat16* r = p.residual + (size_t)ra * p.ldo + cb0;
              if (full) {
#pragma unroll
                for (int j = 0; j < CH / 8; ++j) {
                  const uint4 rr = reinterpret_cast<const uint4*>(r)[j];
                  const uint32_t rw[4] = {rr.x, rr.y, rr.z, rr.w};
#pragma unroll
                  for (int q = 0; q < 4; ++q) {
                    const uint32_t acc = pack_bf16(__uint_as_float(v[8 * j + 2 * q]), __uint_as_float(v[8 * j + 2 * q + 1]));
                    w[4 * j + q] = pack_bf16(bf16_lo(acc) + bf16_lo(rw[q]), bf16_hi(acc) + bf16_hi(rw[q]));
                  }
                }
              } else {
                for (int j = 0; j < CH; ++j)
                  if (cb0 + j < p.Rb)
                    o[j] = __float2bfloat16(__bfloat162float(__float2bfloat16(__uint_as_float(v[j]))) +
                                            __bfloat162float(r[j]));
              }
            } else {
#pragma unroll
              for (int j = 0; j < CH / 2; ++j) w[j] = pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
            }
            if (full) {
#pragma unroll
              for (int j = 0; j < CH / 8; ++j)
                reinterpret_cast<uint4*>(o)[j] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
            } else if constexpr (EPI != EPI_RESIDUAL) {
              for (int j = 0; j < CH; ++j)
                if (cb0 + j < p.Rb) o[j] = reinterpret_cast<__nv_bfloat16*>(w)[j];
            }
          }
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(tempty_bar(as));
    }
  }

  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0) gemm_stamp(p, 9);
  if (warp == 2) tc::tmem_dealloc(tmem_base, TMEM_COLS);
}

static unsigned long long* g_gemm_trace = nullptr;

constexpr uint32_t gemm_stage_bytes(int bn) { return (GEMM_BM + bn) * GEMM_BK * 2; }
constexpr size_t gemm_smem(int stages, int bn) { return (size_t)stages * gemm_stage_bytes(bn) + 8 * (2 * stages + 4) + 16 + 1024; }

template <int BN, int EPI, bool OUT_F32>
static int launch_gemm(const void* a, const void* b, const GemmParams& p0, int Ra, int Rb, int K, int num_sms,
                       cudaStream_t stream) {
  GemmParams p = p0;
  p.trace = g_gemm_trace;
  // whole pieces of 32 columns are stored and read 16 bytes at a time; narrower results go element by element and start anywhere
  JL_CHECK_ARG(Rb < 32 || (((uintptr_t)p.out | (uintptr_t)p.residual) & 15) == 0,
               "jl_gemm: result and residual of the token-major kernel start on a 16-byte boundary (N=%d)", Rb);
  CUtensorMap ta, tb;
  int rc = make_tmap_2d_bf16(&ta, a, Ra, K, K, GEMM_BM);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tb, b, Rb, K, K, BN);
  if (rc) return rc;
  constexpr uint32_t STAGE_BYTES = gemm_stage_bytes(BN);
  const int num_kb = (K + GEMM_BK - 1) / GEMM_BK;
  p.a_blocks = (Ra + GEMM_BM - 1) / GEMM_BM;
  p.b_blocks = (Rb + BN - 1) / BN;
  int grid = p.a_blocks * p.b_blocks;
  if (grid > num_sms) grid = num_sms;
  const int budget = 200 * 1024;
  int stages = (int)(budget / STAGE_BYTES);
  if (stages > 10) stages = 10;
  if (stages > num_kb * 2) stages = num_kb * 2 < 2 ? 2 : num_kb * 2;
  p.stages = stages;
  const size_t smem = gemm_smem(stages, BN);
  auto kern = gemm_kernel<BN, EPI, OUT_F32>;
  JL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  JL_CUDA(launch_pdl(kern, dim3(grid), dim3(GEMM_THREADS), smem, stream, ta, tb, p));
  return JL_OK;
}

template <int EPI, bool OUT_F32>
static int dispatch_gemm(const void* x, const void* w, const GemmParams& p, int M, int N, int K, int num_sms,
                         cudaStream_t s) {
  GemmParams q = p;
  q.Ra = M; q.Rb = N;
  q.hint_a = tc::EVICT_LAST; q.hint_b = tc::EVICT_NORMAL;
  if (N >= 256) return launch_gemm<256, EPI, OUT_F32>(x, w, q, M, N, K, num_sms, s);
  return launch_gemm<128, EPI, OUT_F32>(x, w, q, M, N, K, num_sms, s);
}

}  // namespace jl

using namespace jl;

// Allows (or, with ws == NULL, forbids) split-K on the CURRENT device.  The partials meet in distributed shared memory: the scratch and
// the tickets are not touched.
// Optional timeline of the single-CTA kernel: [grid][16] u64 device buffer (0 entry, 1 set-up done, 2 producer past
// the dependency wait, 3 first stage landed, 4 last MMA issued, 5 accumulator complete, 6 partial published,
// 7 all splits arrived, 8 share emitted, 9 exit); NULL switches it off.
extern "C" JL_API void jl_gemm_set_trace(void* buf) { g_gemm_trace = (unsigned long long*)buf; }

extern "C" JL_API int jl_gemm_set_workspace(void* ws, size_t ws_bytes, int* tickets, int n_tickets) {
  int dev = 0;
  JL_CUDA(cudaGetDevice(&dev));
  JL_CHECK_ARG(dev >= 0 && dev < 16, "jl_gemm_set_workspace: device %d out of range", dev);
  (void)ws_bytes; (void)tickets; (void)n_tickets;
  gemm_swap_allow_split(dev, ws != nullptr);
  return JL_OK;
}

extern "C" JL_API int jl_gemm(const void* x, const void* w, const void* residual, void* out, int M, int N, int K,
                       int mode, int out_f32, int num_sms, void* stream) {
  JL_CHECK_ARG(M >= 1 && N >= 1 && K >= 8 && K % 8 == 0, "jl_gemm: bad shape M=%d N=%d K=%d (K %% 8 == 0)", M, N, K);
  JL_CHECK_ARG(mode >= 0 && mode <= 2, "jl_gemm: bad mode %d", mode);
  JL_CHECK_ARG(mode != EPI_SWIGLU || N % 2 == 0, "jl_gemm: SwiGLU needs an even N");
  JL_CHECK_ARG(mode != EPI_RESIDUAL || residual != nullptr, "jl_gemm: residual pointer missing");
  JL_CHECK_ARG(!(out_f32 && mode != EPI_PLAIN), "jl_gemm: fp32 output only in plain mode");
  JL_CHECK_ARG(N % 8 == 0, "jl_gemm: N=%d must be a multiple of 8", N);
  if (num_sms <= 0) num_sms = 148;
  GemmParams p{};
  p.out = out;
  p.residual = (const __nv_bfloat16*)residual;
  p.K = K;
  p.ldo = mode == EPI_SWIGLU ? N / 2 : N;
  auto s = (cudaStream_t)stream;
  const bool aligned = (((uintptr_t)out | (uintptr_t)residual) & 15) == 0;      // what the token-major kernel wants
  if (out_f32 && gemm_turned_takes(M, N, K, num_sms, aligned)) return gemm_turned_f32(x, w, out, M, N, K, num_sms, g_gemm_trace, s);
  if (gemm_swap_takes(M, N, K, num_sms, aligned)) return gemm_swap(x, w, residual, out, M, N, K, mode, out_f32 != 0, num_sms, g_gemm_trace, s);
  // token-major tiles of the prefill shapes go to the CTA-pair kernel (cta_group::2, gemm_2cta.cu); JLLAMA_GEMM_2CTA=0
  // keeps everything on the single-CTA kernel below (A/B measurements)
  static const bool pair_on = [] { const char* e = getenv("JLLAMA_GEMM_2CTA"); return !(e && e[0] == '0'); }();
  if (pair_on && out_f32 && M >= 256) {
    const int rc = gemm_2cta_f32(x, w, out, M, N, K, num_sms, stream);
    if (rc != JL_ERR_UNSUPPORTED) return rc;
  }
  if (pair_on && !out_f32 && M >= 256) {
    const int rc = jl_gemm_2cta(x, w, residual, out, M, N, K, mode, num_sms, stream);
    if (rc != JL_ERR_UNSUPPORTED) return rc;
  }
  if (mode == EPI_PLAIN && out_f32) return dispatch_gemm<EPI_PLAIN, true>(x, w, p, M, N, K, num_sms, s);
  if (mode == EPI_PLAIN) return dispatch_gemm<EPI_PLAIN, false>(x, w, p, M, N, K, num_sms, s);
  if (mode == EPI_RESIDUAL) return dispatch_gemm<EPI_RESIDUAL, false>(x, w, p, M, N, K, num_sms, s);
  return dispatch_gemm<EPI_SWIGLU, false>(x, w, p, M, N, K, num_sms, s);
}

// bf16 GEMM of few tokens (decode batches, short prompts) on 5th-generation tensor cores: out[M, N] = x[M, K] · W[N, K]^T, M <= 256.
//
// The weights are the MMA's A operand (their rows fill its 128 lanes), the tokens, padded to a multiple of 16, its N: the accumulator is
// the transposed output tile.  Bound by the weight stream.
//   * TMA fills a ring of 64-k stages (128-byte swizzle), one thread issues tcgen05.mma; sums leave TMEM through shared memory as
//     [token][feature], so that a thread stores four neighbouring features of a token (a 2-byte store per lane and token took 8 us of the
//     53 us of 100 x 28672 x 4096);
//   * two CTAs share an SM (half of its shared memory each): up to 296 tiles of 128 weight rows stream at once and end together, where one
//     persistent CTA per SM took 224 tiles in two rounds, the second half empty.  More tiles: the same CTAs walk the list;
//   * few tiles: the CTAs of a cluster of `ksplit` share one and take a part of K each; the finished ring takes the fp32 partial, partials
//     meet in distributed shared memory, each CTA sums its share of the tokens in rank order — deterministic, no scratch in global memory;
//   * up to 128 tokens W is a parameter, which no kernel ahead writes (jllama_b200.h): the ring is filled before the wait for them.  Not above, where W may be any
//     kernel's result (a layer's four products of 129 to 256 tokens: 44.3 us with, 44.9 without at width 1024, 76.4 and 76.8 at 4096), and not in the turned form,
//     whose A operand is the tokens: the kernels ahead let this one start before they have written a row.
// Epilogues: plain bf16 / fp32, residual add, SwiGLU over interleaved (w1, w3) output features.
// One B200, us in a chain of cold weights, one persistent CTA per SM -> this (tokens x features x K): 16 x 28672 x 4096 45.8 -> 38.3 (6.1 TB/s), 16 x
// 24000 x 2048 25.0 -> 17.8, 16 x 11008 x 4096 22.5 -> 18.4, 100 x 28672 x 4096 55 -> 44.5, 100 x 4096 x 4096 17.0 -> 14.1, 100 x 4096 x 14336 34.4 -> 27.8, 128 x 14336 x
// 2048 26.0 -> 16.2; 16 x 128256 x 2048 81.6 -> 81.3.
//
// The linear layers of jax_llama/model.py:119-150, :311-338 and :699-706 at decode and for short prompts.
#include <atomic>
#include <type_traits>

#include "gemm_swap.cuh"
#include "jllama_b200.h"
#include "tcgen05.cuh"

namespace jl {

constexpr int GS_BM = 128, GS_BK = 64, GS_THREADS = 256;        // warp 0: TMA, warp 1: MMA, warp 2: TMEM; all: epilogue
constexpr uint32_t GS_A_BYTES = GS_BM * GS_BK * 2, GS_STAGING = 16 * GS_BM * 4;

struct SwapParams {
  void* out;
  const __nv_bfloat16* residual;
  int N, M, K, nb;          // weight rows, tokens, reduction length, tokens padded to a multiple of 16
  int ldo, stages, ksplit, wide;   // wide: out and residual take 4-feature accesses
  int turned;                      // the A operand is the tokens and the result's rows are its rows (fp32): out[feature * ldo + token]; nothing is asked for early
  uint32_t cols, idesc;
  unsigned long long* trace;       // optional [trace_rows][16] %globaltimer stamps (jl_gemm_set_trace), NULL = off
  int trace_rows;
};

// one thread records when it reached a point of the kernel (scripts/gemm_trace.py prints the timeline)
__device__ __forceinline__ void swap_stamp(const SwapParams& p, int ev) {
  if (p.trace != nullptr && (int)blockIdx.x < p.trace_rows) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t)::"memory");
    p.trace[(size_t)blockIdx.x * 16 + ev] = t;
  }
}

__device__ __forceinline__ void swap_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void swap_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t swap_mapa(uint32_t local_addr, int rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local_addr), "r"(rank));
  return a;
}
__device__ __forceinline__ float4 swap_ld_cluster(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
constexpr int GS_LINES = 160;                            // floats of a token's partial as lines: four of 32, 40 apart
__device__ __forceinline__ float4 swap_ld_lines(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v.x) : "r"(addr) : "memory");
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v.y) : "r"(addr + 160) : "memory");
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v.z) : "r"(addr + 320) : "memory");
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v.w) : "r"(addr + 480) : "memory");
  return v;
}

// residual of four neighbouring features of a token
__device__ __forceinline__ uint2 swap_residual(const SwapParams& p, int tok, int f0) {
  const __nv_bfloat16* r = p.residual + (size_t)tok * p.ldo + f0;
  if (p.wide) return *reinterpret_cast<const uint2*>(r);
  const unsigned short* h = reinterpret_cast<const unsigned short*>(r);
  return make_uint2(h[0] | (uint32_t)h[1] << 16, h[2] | (uint32_t)h[3] << 16);
}
// finish and store four neighbouring features of a token
template <int EPI, bool OUT_F32>
__device__ __forceinline__ void swap_emit(const SwapParams& p, int tok, int f0, const float (&x)[4], uint2 res) {
  if constexpr (OUT_F32) {
    if (p.turned) {
      float* o = reinterpret_cast<float*>(p.out) + (size_t)f0 * p.ldo + tok;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (f0 + i < p.N) o[(size_t)i * p.ldo] = x[i];
      return;
    }
    float* o = reinterpret_cast<float*>(p.out) + (size_t)tok * p.ldo + f0;
    if (p.wide) *reinterpret_cast<float4*>(o) = make_float4(x[0], x[1], x[2], x[3]);
    else { o[0] = x[0]; o[1] = x[1]; o[2] = x[2]; o[3] = x[3]; }
    return;
  }
  uint32_t a = pack_bf16(x[0], x[1]), b = pack_bf16(x[2], x[3]);
  if constexpr (EPI == SWAP_SWIGLU) {
    const uint32_t y = pack_bf16(silu(bf16_lo(a)) * bf16_hi(a), silu(bf16_lo(b)) * bf16_hi(b));
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)tok * p.ldo + f0 / 2;
    if (p.wide) *reinterpret_cast<uint32_t*>(o) = y;
    else { reinterpret_cast<unsigned short*>(o)[0] = (unsigned short)y; reinterpret_cast<unsigned short*>(o)[1] = (unsigned short)(y >> 16); }
  } else {
    if constexpr (EPI == SWAP_RESIDUAL) {
      a = pack_bf16(bf16_lo(a) + bf16_lo(res.x), bf16_hi(a) + bf16_hi(res.x));
      b = pack_bf16(bf16_lo(b) + bf16_lo(res.y), bf16_hi(b) + bf16_hi(res.y));
    }
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)tok * p.ldo + f0;
    if (p.wide) *reinterpret_cast<uint2*>(o) = make_uint2(a, b);
    else {
      unsigned short* h = reinterpret_cast<unsigned short*>(o);
      h[0] = (unsigned short)a; h[1] = (unsigned short)(a >> 16); h[2] = (unsigned short)b; h[3] = (unsigned short)(b >> 16);
    }
  }
}

template <int EPI, bool OUT_F32, bool SPLIT>
__global__ void __launch_bounds__(GS_THREADS, 2)
gemm_swap_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const SwapParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (tc::smem_u32(smem_raw) + 1023u) & ~1023u;
  const int stages = p.stages, ksplit = SPLIT ? p.ksplit : 1;
  const uint32_t b_bytes = (uint32_t)p.nb * (GS_BK * 2), stage_bytes = GS_A_BYTES + b_bytes;
  const uint32_t staging = smem_base + stages * stage_bytes;    // !SPLIT: 16 tokens x 32 features fp32 for each epilogue warp
  const uint32_t bars = staging + (SPLIT ? 0u : GS_STAGING);      // full[stages] | empty[stages] | tfull[2] | tempty[2]
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (stages + s); };
  auto tfull_bar = [&](int s) { return bars + 8u * (2 * stages + s); };
  auto tempty_bar = [&](int s) { return bars + 8u * (2 * stages + 2 + s); };
  const uint32_t tmem_slot = bars + 8u * (2 * stages + 4);
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - tc::smem_u32(smem_raw)));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_kb = (p.K + GS_BK - 1) / GS_BK, tiles = (p.N + GS_BM - 1) / GS_BM;
  const int tile0 = (int)blockIdx.x / ksplit, tstep = (int)gridDim.x / ksplit;      // SPLIT: one tile, its parts are the CTAs of a cluster
  const int rank = (int)blockIdx.x % ksplit, kb0 = rank * num_kb / ksplit, kb1 = (rank + 1) * num_kb / ksplit;

  if (threadIdx.x == 0) swap_stamp(p, 0);
  if (warp == 0 && lane == 0) {
    tc::prefetch_tensormap(&tmap_w);
    tc::prefetch_tensormap(&tmap_x);
  }
  if (warp == 1 && lane == 0) {
    for (int s = 0; s < stages; ++s) { tc::mbar_init(full_bar(s), 1); tc::mbar_init(empty_bar(s), 1); }
    for (int s = 0; s < 2; ++s) { tc::mbar_init(tfull_bar(s), 1); tc::mbar_init(tempty_bar(s), 4); }
    tc::fence_barrier_init();
  }
  if (warp == 2) tc::tmem_alloc(tmem_slot, SPLIT ? p.cols : 2 * p.cols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = *tmem_slot_ptr;
  // The next kernel of the chain may start: it waits for this grid itself before it touches anything this grid writes, and ITS weight prefetch (below)
  // overlaps our epilogue.  Not before this CTA has its columns of tensor memory: a kernel that takes all 512 ahead of its wait would keep them until this
  // grid is done, and this grid would wait for them.  (At the top of the kernel: the smallest sizes 0.1 us faster, 5 x 1024 x 1024 4.2 and 4.35.)
  pdl_launch_dependents();
  if (threadIdx.x == 0) swap_stamp(p, 1);

  if (warp == 0) {
    // ===================================================== TMA producer
    if (lane == 0) {
      // weights stream from HBM while the previous kernel runs its tail; the tokens follow after the wait for it
      int pre = p.turned || p.M > 128 ? 0 : kb1 - kb0 < stages ? kb1 - kb0 : stages;
      const uint64_t hint_a = p.turned ? tc::EVICT_NORMAL : tc::EVICT_FIRST;      // (tokens are read again by the kernels behind)
      for (int i = 0; i < pre; ++i) {
        tc::mbar_expect_tx(full_bar(i), stage_bytes);
        tc::tma_load_2d(smem_base + i * stage_bytes, &tmap_w, full_bar(i), (kb0 + i) * GS_BK, tile0 * GS_BM, hint_a);
      }
      pdl_wait();
      swap_stamp(p, 2);
      int stage = 0; uint32_t phase = 0;
      for (int tile = tile0; tile < tiles; tile += tstep) {
        for (int kb = kb0; kb < kb1; ++kb) {
          const uint32_t sa = smem_base + stage * stage_bytes;
          if (pre > 0) {
            --pre;
          } else {
            tc::mbar_wait(empty_bar(stage), phase ^ 1);
            tc::mbar_expect_tx(full_bar(stage), stage_bytes);
            tc::tma_load_2d(sa, &tmap_w, full_bar(stage), kb * GS_BK, tile * GS_BM, hint_a);
          }
          tc::tma_load_2d(sa + GS_A_BYTES, &tmap_x, full_bar(stage), kb * GS_BK, 0, tc::EVICT_LAST);
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ===================================================== MMA issuer (single thread)
    if (lane == 0) {
      int stage = 0, it = 0; uint32_t phase = 0;
      for (int tile = tile0; tile < tiles; tile += tstep, ++it) {
        const int as = it & 1;
        if constexpr (!SPLIT) {
          tc::mbar_wait(tempty_bar(as), ((it >> 1) & 1) ^ 1);      // the epilogue has drained this accumulator
          tc::fence_after_sync();
        }
        const uint32_t d = tmem_base + as * p.cols;
        for (int kb = kb0; kb < kb1; ++kb) {
          tc::mbar_wait(full_bar(stage), phase);
          tc::fence_after_sync();
          if (it == 0 && kb == kb0) swap_stamp(p, 3);
          const uint32_t sa = smem_base + stage * stage_bytes;
          const uint64_t da = tc::smem_desc_kmajor_sw128(sa), db = tc::smem_desc_kmajor_sw128(sa + GS_A_BYTES);
#pragma unroll
          for (int k = 0; k < GS_BK / 16; ++k)              // +32 bytes per UMMA_K inside the swizzle span
            tc::mma_ss(d, da + 2 * k, db + 2 * k, p.idesc, kb != kb0 || k != 0);
          tc::mma_commit(empty_bar(stage));                 // frees the smem slot when these MMAs retire
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
        tc::mma_commit(tfull_bar(as));
        if (it == 0) swap_stamp(p, 4);
      }
    }
    __syncwarp();
  }

  // TMEM lane = weight row, column = token.  Sums go through shared memory as [token][feature] and come back four features of a token to
  // a thread.
  const uint32_t t_lane = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
  auto to_shared = [&](uint32_t t_col, uint32_t at, int pitch) {      // 16 tokens
    uint32_t v[16];
    tc::tmem_ld16(t_col, v);
    tc::tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + j * pitch), "r"(v[j]) : "memory");
  };
  if constexpr (!SPLIT) {
    // ===================================================== epilogue of a persistent CTA: warps 4-7, 16 tokens at a time
    if (warp >= 4) {
      pdl_wait();                                           // residual, output: after the previous kernel
      const uint32_t st = staging + (warp & 3) * (GS_STAGING / 4);
      int it = 0;
      for (int tile = tile0; tile < tiles; tile += tstep, ++it) {
        const int as = it & 1, f0 = tile * GS_BM + (warp & 3) * 32 + 4 * (lane & 7);      // N % 4 == 0: all four features are inside or none
        tc::mbar_wait(tfull_bar(as), (it >> 1) & 1);
        tc::fence_after_sync();
        if (it == 0 && threadIdx.x == 128) swap_stamp(p, 5);
        for (int c0 = 0; c0 < p.nb; c0 += 16) {
          uint2 res[4];
          if constexpr (EPI == SWAP_RESIDUAL) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int tok = c0 + (lane >> 3) + 4 * u;
              res[u] = f0 < p.N && tok < p.M ? swap_residual(p, tok, f0) : make_uint2(0u, 0u);
            }
          }
          to_shared(t_lane + as * p.cols + c0, st + lane * 4, 128);
          tc::fence_before_sync();
          __syncwarp();
          if (c0 + 16 >= p.nb && lane == 0) tc::mbar_arrive(tempty_bar(as));      // read: the sums of the tile after next may begin
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int row = (lane >> 3) + 4 * u, tok = c0 + row;
            if (f0 >= p.N || tok >= p.M) continue;
            float x[4];
            asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(st + row * 128 + (lane & 7) * 16) : "memory");
            swap_emit<EPI, OUT_F32>(p, tok, f0, x, res[u]);
          }
          __syncwarp();
        }
        if (it == 0 && threadIdx.x == 128) swap_stamp(p, 8);
      }
    }
  } else {
    // ===================================================== all warps: partial sums meet in the cluster
    pdl_wait();
    const int f0 = tile0 * GS_BM + 4 * lane;                // a warp writes 256 (SwiGLU: 128) contiguous bytes of a token
    // A token's partial: its features in a row, read 16 bytes a lane, four ranks' four tokens at once; or feature 4 l + j at 40 j + l, read as four lines of
    // 128 bytes, all ranks' one token at once (the pitch of 40 keeps the writes off one another's banks).  From four ranks on the lines are faster, since a warp's
    // 512 bytes of another SM's memory come in four pieces either way; with two or three ranks they leave too little in flight.  Rows -> lines, us: 16 x 2048 x 2048, 8
    // ranks, 5.24 -> 5.08; 5 x 1024 x 2048, 8 ranks, 4.8 -> 4.2; 128 x 3072 x 2048, 6 ranks, 12.3 -> 10.9; 128 x 4096 x 2048, 4 ranks, 11.4 -> 10.5; 128 x 8192 x 2048, 2 ranks,
    // 12.8 -> 14.2; 256 x 6144 x 2048, 3 ranks, 14.9 -> 18.3; and 128 x 1024 x 14336, 16 ranks, 17.0 -> 17.9 (100 tokens 15.8 and 15.7).
    const bool lines = ksplit >= 4 && (ksplit <= 8 || p.nb <= 112);
    const int row = lines ? GS_LINES * 4 : GS_BM * 4;
    const uint32_t put = smem_base + (lines ? (lane & 3) * 40 + (warp & 3) * 8 + lane / 4 : (warp & 3) * 32 + lane) * 4, get = smem_base + lane * (lines ? 4 : 16);
    const bool on = f0 < p.N;
    const int per = (p.M + ksplit - 1) / ksplit, t_lo = rank * per, t_hi = t_lo + per < p.M ? t_lo + per : p.M;
    uint2 res[4];
    auto load_res = [&](int tok0, int n) {                  // residual of n tokens from tok0 in steps of eight
      if constexpr (EPI == SWAP_RESIDUAL) {
#pragma unroll
        for (int u = 0; u < 4; ++u) if (u < n) res[u] = on && tok0 + 8 * u < t_hi ? swap_residual(p, tok0 + 8 * u, f0) : make_uint2(0u, 0u);
      }
    };
    load_res(t_lo + warp, lines ? 1 : 4);
    tc::mbar_wait(tfull_bar(0), 0);
    tc::fence_after_sync();
    if (threadIdx.x == 128) swap_stamp(p, 5);
    // the ring is free (one tile per CTA, all its MMAs done) and takes the partial
    for (int c0 = (warp >> 2) * 16; c0 < p.nb; c0 += 32) to_shared(t_lane + c0, put + c0 * row, row);
    if (threadIdx.x == 128) swap_stamp(p, 6);
    swap_cluster_arrive();
    swap_cluster_wait();
    if (threadIdx.x == 128) swap_stamp(p, 7);
    auto meet = [&](auto ranks, auto tokens) {              // a warp takes a token at a time of each group of `tokens`
      constexpr int R = decltype(ranks)::value, U = decltype(tokens)::value;
      for (int tok0 = t_lo + warp; tok0 < t_hi; tok0 += 8 * U) {
        if (tok0 != t_lo + warp) load_res(tok0, U);
        float x[U][4] = {};
        for (int r0 = 0; r0 < ksplit; r0 += R) {
          float4 q[R][U];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (r0 + r >= ksplit) continue;
            const uint32_t at = swap_mapa(get, r0 + r);
#pragma unroll
            for (int u = 0; u < U; ++u) {
              if (tok0 + 8 * u >= t_hi) continue;
              if constexpr (U == 1) q[r][u] = swap_ld_lines(at + (tok0 + 8 * u) * (GS_LINES * 4));
              else q[r][u] = swap_ld_cluster(at + (tok0 + 8 * u) * (GS_BM * 4));
            }
          }
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (r0 + r >= ksplit) continue;
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (tok0 + 8 * u < t_hi) { x[u][0] += q[r][u].x; x[u][1] += q[r][u].y; x[u][2] += q[r][u].z; x[u][3] += q[r][u].w; }
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (on && tok0 + 8 * u < t_hi) swap_emit<EPI, OUT_F32>(p, tok0 + 8 * u, f0, x[u], res[u]);
      }
    };
    if (lines && ksplit > 8) meet(std::integral_constant<int, 16>{}, std::integral_constant<int, 1>{});
    else if (lines) meet(std::integral_constant<int, 8>{}, std::integral_constant<int, 1>{});
    else meet(std::integral_constant<int, 4>{}, std::integral_constant<int, 4>{});
    if (threadIdx.x == 128) swap_stamp(p, 8);
    swap_cluster_arrive();                                  // no CTA leaves while its partial may still be read
    swap_cluster_wait();
  }
  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0) swap_stamp(p, 9);
  if (warp == 2) tc::tmem_dealloc(tmem_base, SPLIT ? p.cols : 2 * p.cols);
}

// whether the caller allows split-K on a device (jl_gemm_set_workspace)
static bool g_splitk[16] = {};
static bool splitk_allowed() {
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 16 && g_splitk[dev];
}
void gemm_swap_allow_split(int device, bool on) { g_splitk[device] = on; }

constexpr size_t gs_smem(int stages, int nb, bool split) {
  return (size_t)stages * (GS_A_BYTES + nb * GS_BK * 2) + (split ? 0 : GS_STAGING) + 8 * (2 * stages + 4) + 16 + 1024;
}

// ring depth: two CTAs per SM up to 128 tokens; the fp32 partial (up to 640 bytes a token) of a split fits the ring in every case
static int gs_stages(int nb, int num_kb, bool split) {
  const int stage = (int)(GS_A_BYTES + nb * GS_BK * 2), budget = nb > 128 ? 200 * 1024 : 111 * 1024 - (split ? 0 : (int)GS_STAGING);
  int stages = budget / stage;
  if (stages > 10) stages = 10;
  const int tile = split ? (nb * GS_LINES * 4 + stage - 1) / stage : 2;
  if (stages > num_kb) stages = num_kb;
  return stages < tile ? tile : stages;
}

// whether the device holds clusters of `ks` > 8 CTAs of the split-K kernel (asked once per device, kernel and size)
template <int EPI, bool OUT_F32>
static bool wide_clusters(int ks, int num_sms) {
  static std::atomic<signed char> known[16][17];          // 0: not asked yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return false;
  signed char v = known[dev][ks].load(std::memory_order_relaxed);
  if (v == 0) {
    auto kern = gemm_swap_kernel<EPI, OUT_F32, true>;
    int n = 0;
    size_t smem = 0;                                       // the largest of all token counts (48: 5 stages of 22 KB, 16: 6 of 18)
    for (int nb = 16; nb <= 128; nb += 16) {
      const size_t s = gs_smem(gs_stages(nb, 1 << 20, true), nb, true);
      if (s > smem) smem = s;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(num_sms / ks * ks);
    cfg.blockDim = dim3(GS_THREADS);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ks; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess &&
                    cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n >= 1;
    if (!ok) cudaGetLastError();
    v = ok ? 1 : -1;
    known[dev][ks].store(v, std::memory_order_relaxed);
  }
  return v > 0;
}

// Parts of K, a cluster's CTAs.  At least 4 k-blocks (256 columns) per CTA; enough parts to give every SM one CTA, and more, up to what
// the two slots of an SM hold, while a part keeps 16 k-blocks.  Clusters of 3 to 8 find place for 264 CTAs (288: a second round, 48 tiles in 6 parts
// 17.8 us, in 4 12.6), pairs for 2 x SMs.  16 tokens, us: 32 tiles, K 14336: 4 parts 24.1, 8 22.9; 86 tiles, K 4096: 1 part 23.3, 2 18.7, 3 18.4; 112
// tiles 1 24.8, 2 22.1; 128 tokens: 32 x 14336 33.4 -> 29.6, 86 x 4096 31.0 -> 21.7, 112 x 4096 34.0 -> 25.3; shorter parts give nothing (32 tiles, K 4096, 4 parts
// 10.6, 8 10.4; 128 tokens 15.5 and 15.7).  Pairs that fill both slots of nearly every SM have to have longer parts where the tokens are few (16 tokens, 148 tiles: K 2048
// 1 part 15.2, 2 16.2, K 3072 22.1 and 22.2; 133 tiles, K 4096 27.8 and 25.1; 64 tokens, 148 tiles, K 2048 16.5 and 16.5).
// Eight CTAs are what every GPU takes as a cluster.  More pay with a long K over few tiles (9 to 16 rows of 1024 x 14336: 8 parts 11.8 us, 16
// parts 10.1; 1536 x 14336 12.8 and 12.0 in 12 parts); at K 8192 and below, and with less than half as many again, the wider meeting costs
// what it gives or more (1024 x 4096 5.8 and 5.9 us, 64 rows 7.8 and 8.5; 2048 x 14336, 9 parts, 13.7 and 14.1).
// Above 128 tokens a CTA fills an SM: clusters of up to 4 (200 tokens: 16 tiles in 4 parts 9.8 us, in 8 19.6; 48 tiles in 2 parts 18.7, in 3 29.7).
template <int EPI, bool OUT_F32>
static int swap_parts(int nb, int tiles, int num_kb, int num_sms) {
  if (!splitk_allowed()) return 1;
  int ks = num_sms / tiles;
  if (nb > 128) {
    if (ks > 4) ks = 4;
    while (ks > 2 && tiles * ks > num_sms - 20) --ks;
  } else {
    if (ks > 16) ks = 16;
    if (ks > 8 && (ks < 12 || num_kb <= 128 || !wide_clusters<EPI, OUT_F32>(ks, num_sms))) ks = 8;
    int more = num_kb / 16 < 8 ? num_kb / 16 : 8;
    while (more > 2 && tiles * more > 2 * num_sms - 32) --more;
    if (more == 2 && (tiles > num_sms || (nb <= 32 && tiles > num_sms - 16 && num_kb < 48))) more = 1;
    if (more > ks) ks = more;
  }
  if (ks > num_kb / 4) ks = num_kb / 4;
  return ks > 1 ? ks : 1;
}

template <int EPI, bool OUT_F32>
static int launch_swap(const void* x, const void* w, const void* residual, void* out, int M, int N, int K, int num_sms,
                       unsigned long long* trace, cudaStream_t stream, bool turned = false) {
  SwapParams p{};
  p.out = out;
  p.residual = (const __nv_bfloat16*)residual;
  p.N = N; p.M = M; p.K = K;
  p.nb = (M + 15) / 16 * 16;
  p.ldo = turned ? M : EPI == SWAP_SWIGLU ? N / 2 : N;
  p.turned = turned;
  const uintptr_t step = OUT_F32 ? 16 : EPI == SWAP_SWIGLU ? 4 : 8;
  p.wide = (((uintptr_t)out | (uintptr_t)residual) & (step - 1)) == 0;
  p.cols = p.nb <= 32 ? 32 : p.nb <= 64 ? 64 : p.nb <= 128 ? 128 : 256;
  p.idesc = tc::idesc_bf16_f32(GS_BM, p.nb);
  p.trace = trace;
  p.trace_rows = num_sms;
  CUtensorMap tw, tx;
  int rc = make_tmap_2d_bf16(&tw, w, N, K, K, GS_BM);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tx, x, M, K, K, p.nb);
  if (rc) return rc;
  const int num_kb = (K + GS_BK - 1) / GS_BK, tiles = (N + GS_BM - 1) / GS_BM;
  p.ksplit = swap_parts<EPI, OUT_F32>(p.nb, tiles, num_kb, num_sms);
  const bool split = p.ksplit > 1;
  const int slots = p.nb <= 128 ? 2 * num_sms : num_sms;
  p.stages = gs_stages(p.nb, split ? (num_kb + p.ksplit - 1) / p.ksplit : (tiles + slots - 1) / slots * num_kb, split);
  const size_t smem = gs_smem(p.stages, p.nb, split);
  auto kern = split ? gemm_swap_kernel<EPI, OUT_F32, true> : gemm_swap_kernel<EPI, OUT_F32, false>;
  JL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(split ? tiles * p.ksplit : tiles < slots ? tiles : slots);
  cfg.blockDim = dim3(GS_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (split) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = p.ksplit;
    attr[na].val.clusterDim.y = 1;
    attr[na++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  count_launch();
  JL_CUDA(cudaLaunchKernelEx(&cfg, kern, tw, tx, p));
  return JL_OK;
}

// Up to 128 tokens always; up to 256 where K can be split over a cluster: the token-major kernel has (M / 128) x (N / 256) tiles there and no
// split (200 tokens, us: 4096 x 4096 31.1 -> 14.5, 4096 x 14336 90.8 -> 30.6, 6144 x 4096 30.0 -> 18.7, 2048 x 2048 18.9 -> 9.8, 1024 x 1024 8.9 -> 7.7); with more
// weights the two are equal (28672 x 4096: 62 us).  What a split costs more the tokens and the tile of few features have to earn: of 256 and more features it pays from K 512
// (200 tokens x 512, K 512: fp32 9.3 -> 7.6 us, bfloat16 6.7 -> 7.1), above 200 tokens from 768 (256 x 256, fp32: K 512 6.9 -> 7.8, 768 7.9 -> 8.3, 1024 9.1 -> 8.9;
// bfloat16, K 768 9.5 -> 7.9), of fewer from 1024 (200 x 128, K 1024: fp32 8.5 -> 8.0, bfloat16 7.2 -> 7.6; K 768, bfloat16 6.2 -> 6.9) or 1536 (256 x 128, bfloat16: K 1024 7.3 -> 8.1,
// 2048 11.6 -> 9.7).  A result or residual off the 16-byte boundary comes here at every size.
bool gemm_swap_takes(int M, int N, int K, int num_sms, bool aligned) {
  if (M <= 128) return true;
  const int from = !aligned ? 8 * GS_BK : N >= 256 ? (M <= 200 ? 512 : 768) : (M <= 200 ? 1024 : 1536);
  return M <= 256 && (N + GS_BM - 1) / GS_BM * 2 <= num_sms && K >= from && splitk_allowed();
}

// Few output features over many tokens (a router): the tokens take the MMA's rows, 128 to a tile, and K is split over clusters, where the token-major kernel has a
// tile, i.e. a CTA, per 128 tokens.  Nothing is asked for ahead of the wait.  Token-major -> this, us a launch in a chain of cold tokens (32 features, K 2048): 512 tokens
// 12.1 -> 6.0, 2048 12.3 -> 7.2, 4096 12.4 -> 8.8; 64 features, K 4096, 2048 tokens 21.6 ->
// 10.4; what it adds behind the norm that writes its tokens: 2048 tokens 11.7 -> 6.6 us.  The line in K, norm and product of 512 tokens: 16 features, K 512 7.8 -> 6.8; 32, K 512 7.2
// -> 7.6, 768 8.7 -> 7.3; 64, K 512 7.6 -> 8.9, 768 9.0 -> 8.9, 1024 10.6 -> 8.4.  (Products of that kind alone, one behind the other, overlap better in the token-major
// kernel, which leaves SMs free: 4096 tokens, 64 features, K 1024 7.9 and 9.0.)
bool gemm_turned_takes(int M, int N, int K, int num_sms, bool aligned) {
  const int from = !aligned || N <= 16 ? 512 : N <= 32 ? 768 : 1024;
  return N <= 64 && M > 128 && (M + GS_BM - 1) / GS_BM * 4 <= num_sms && K >= from && splitk_allowed();
}
int gemm_turned_f32(const void* x, const void* w, void* out, int M, int N, int K, int num_sms, unsigned long long* trace, cudaStream_t s) {
  return launch_swap<SWAP_PLAIN, true>(w, x, nullptr, out, N, M, K, num_sms, trace, s, true);
}

int gemm_swap(const void* x, const void* w, const void* residual, void* out, int M, int N, int K, int mode, bool out_f32, int num_sms,
              unsigned long long* trace, cudaStream_t s) {
  if (mode == SWAP_PLAIN && out_f32) return launch_swap<SWAP_PLAIN, true>(x, w, nullptr, out, M, N, K, num_sms, trace, s);
  if (mode == SWAP_PLAIN) return launch_swap<SWAP_PLAIN, false>(x, w, nullptr, out, M, N, K, num_sms, trace, s);
  if (mode == SWAP_RESIDUAL) return launch_swap<SWAP_RESIDUAL, false>(x, w, residual, out, M, N, K, num_sms, trace, s);
  return launch_swap<SWAP_SWIGLU, false>(x, w, nullptr, out, M, N, K, num_sms, trace, s);
}

}  // namespace jl

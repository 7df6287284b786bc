// Prompt attention on tcgen05 for the head shapes of the generic kernels: query / key rows of 64, 128, 192 or 256 channels, value rows
// of 64 or 128, any row pitch and batch / head strides (per-head caches, token-major projections), bfloat16.
//
// attn_rows_kernel (attn_generic.cu) keeps scores, probabilities and sums in fp32, and so does this kernel: a probability goes to the
// tensor core as TWO bfloat16 numbers, hi + lo = p to 2^-17, and P·V is two products into the same fp32 accumulator.  (The plain flash
// kernel, flash_prefill.cu, rounds p to one bfloat16.)  Rounded to bfloat16 are the inputs and the output, as before; the tensor core's sums cut
// off where an FMA rounds, and p has 17 bits instead of 24.  What that is in the result, against float64, attn_rows_kernel -> this one (2-norm, over
// four draws; D / Dv, tokens): 192 / 128, 2048, window 1024 1.69910e-3 -> 1.69910e-3; the same without a window and scores four times as
// large 1.65928e-3 -> 1.65928e-3; 64 / 64, 700 1.68426e-3 -> 1.68426e-3: the output's rounding, in which one result of a thousand falls the other way.
//
// One CTA per 128 queries of one head, six warps: a TMA warp (Q once; K and V tiles of 64 keys through two-slot rings), an MMA warp,
// four softmax warps with one query row per thread.
//   S = Q·Kᵀ   D / 16 MMAs of 128 x 64 x 16 into one of two score tiles in TMEM, the next tile's issued before this one is consumed;
//   softmax    as in flash_prefill.cu: one pass over the row's 64 scores in registers, a lazily raised reference maximum, O rescaled
//              in TMEM only when the maximum has grown by 2^8; the 64 score columns are overwritten by hi (32 columns of packed pairs) and
//              lo (32 columns);
//   O += P·V   eight MMAs per tile, A from TMEM.
// Slots that no query of the CTA sees (behind the last key, before the first one) may hold anything: their scores are masked, and the softmax
// warps clear their value rows in shared memory, because a weight of zero times a NaN is a NaN.
// Bound: per tile 64 · D + 2 · 64 · Dv MACs of a row against 64 exponentials; at D 192, Dv 128 the tensor work is 900 cycles, the
// softmax warps need about as many.  2048 tokens, 16 heads, D 192, Dv 128, window 1024 on one B200: 41 us; attn_rows_kernel 1173 us
// (fp32 FMAs from shared memory).
#include "flash_wide.cuh"
#include "jllama_b200.h"
#include "seq_types.cuh"
#include "tcgen05.cuh"

namespace jl {

constexpr int FW_BM = 128, FW_BN = 64, FW_THREADS = 192, FW_SLOTS = 2;
constexpr uint32_t FW_Q_CHUNK = FW_BM * 128, FW_KV_CHUNK = FW_BN * 128;      // bytes of 64 channels of a tile's rows
constexpr float FW_RESCALE = 8.0f;                                          // log2 units

__host__ __device__ constexpr uint32_t fw_tiles_bytes(int kc, int vc) { return kc * FW_Q_CHUNK + FW_SLOTS * (kc + vc) * FW_KV_CHUNK; }
__host__ __device__ constexpr uint32_t fw_smem_bytes(int kc, int vc) { return fw_tiles_bytes(kc, vc) + 1024 + 128; }

__device__ __forceinline__ void fw_tma_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4, %5, %6}], [%2], %7;" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "l"(tc::EVICT_NORMAL)
      : "memory");
}

// 2^x with exp2f's error, but results below 2^-126 are zero (nothing beside a maximum of at least 2^-8): what exp2f does for these made
// the kernel 4 to 13 % slower (2048 tokens, 16 heads: 192 / 128 channels 40.4 -> 42.1 us, 64 / 64 35.5 -> 40.0)
__device__ __forceinline__ float fw_exp2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// KC / VC: 64-channel chunks of a query / key row and of a value row.
template <int KC, int VC>
__global__ void __launch_bounds__(256, KC <= 2 ? 2 : 1)
flash_wide_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                  const __grid_constant__ CUtensorMap tmap_v, const FlashWide p) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const uint32_t raw = tc::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t sQ = base;
  auto sK = [&](int s) { return base + KC * FW_Q_CHUNK + (uint32_t)s * KC * FW_KV_CHUNK; };
  auto sV = [&](int s) { return base + KC * FW_Q_CHUNK + FW_SLOTS * KC * FW_KV_CHUNK + (uint32_t)s * VC * FW_KV_CHUNK; };
  const uint32_t bars = base + fw_tiles_bytes(KC, VC);
  const uint32_t q_full = bars, p_full = bars + 8, o_full = bars + 16;
  auto k_full = [&](int s) { return bars + 24 + 8u * s; };
  auto k_empty = [&](int s) { return bars + 40 + 8u * s; };
  auto v_full = [&](int s) { return bars + 56 + 8u * s; };
  auto v_empty = [&](int s) { return bars + 72 + 8u * s; };
  auto s_full = [&](int s) { return bars + 88 + 8u * s; };
  const uint32_t tmem_slot = bars + 104;
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - raw));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // longest query tiles first over the whole grid, the heads of a tile next to each other (flash_prefill.cu)
  const int lin = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  const int n_hb = gridDim.y * gridDim.z;
  const int q0 = ((int)gridDim.x - 1 - lin / n_hb) * FW_BM;
  const int h = (lin % n_hb) % (int)gridDim.y, b = (lin % n_hb) / (int)gridDim.y;
  const int g = h / (p.H / p.G);

  if (warp == 0 && lane == 0) {
    tc::prefetch_tensormap(&tmap_q); tc::prefetch_tensormap(&tmap_k); tc::prefetch_tensormap(&tmap_v);
  }
  if (warp == 1 && lane == 0) {
    tc::mbar_init(q_full, 1); tc::mbar_init(p_full, 4); tc::mbar_init(o_full, 1);
    for (int s = 0; s < 2; ++s) {
      tc::mbar_init(k_full(s), 1); tc::mbar_init(k_empty(s), 1); tc::mbar_init(v_full(s), 1); tc::mbar_init(v_empty(s), 1);
      tc::mbar_init(s_full(s), 1);
    }
    tc::fence_barrier_init();
  }
  if (warp == 0) tc::tmem_alloc(tmem_slot, 256);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot_ptr;
  auto tS = [&](int j) { return tmem + (uint32_t)(j & 1) * 64u; };     // score tile j, afterwards hi | lo of its probabilities
  const uint32_t tO = tmem + 128;

  pdl_wait();
  pdl_launch_dependents();

  const int start = p.cache_len ? *p.cache_len : 0;
  const int pad = p.pad_left ? p.pad_left[b] : 0;
  const int q_hi = min(q0 + FW_BM, p.S) - 1;
  auto first_seen = [&](int slot) {                        // first key a query at `slot` sees (grows with the slot)
    int lo = pad;
    if (p.window > 0) lo = max(lo, slot - p.window + 1);
    if (p.chunk > 0 && slot >= pad) lo = max(lo, pad + (slot - pad) / p.chunk * p.chunk);
    return lo;
  };
  const int first_tile = first_seen(start + q0) / FW_BN;
  const int last_tile = (start + q_hi) / FW_BN;
  const int n_tiles = last_tile - first_tile + 1 > 0 ? last_tile - first_tile + 1 : 0;

  if (warp == 0) {
    if (lane == 0) {
      tc::mbar_expect_tx(q_full, KC * FW_Q_CHUNK);
#pragma unroll
      for (int c = 0; c < KC; ++c) fw_tma_4d(sQ + c * FW_Q_CHUNK, &tmap_q, q_full, 64 * c, q0, h, b);
      for (int j = 0; j < n_tiles; ++j) {
        const int sl = j & 1; const uint32_t ph = ((j >> 1) & 1) ^ 1;
        const int key0 = (first_tile + j) * FW_BN;
        tc::mbar_wait(k_empty(sl), ph);
        tc::mbar_expect_tx(k_full(sl), KC * FW_KV_CHUNK);
#pragma unroll
        for (int c = 0; c < KC; ++c) fw_tma_4d(sK(sl) + c * FW_KV_CHUNK, &tmap_k, k_full(sl), 64 * c, key0, g, b);
        tc::mbar_wait(v_empty(sl), ph);
        tc::mbar_expect_tx(v_full(sl), VC * FW_KV_CHUNK);
#pragma unroll
        for (int c = 0; c < VC; ++c) fw_tma_4d(sV(sl) + c * FW_KV_CHUNK, &tmap_v, v_full(sl), 64 * c, key0, g, b);
      }
    }
  } else if (warp == 1) {
    // the whole warp walks the loop, one elected lane issues (flash_prefill.cu)
    constexpr uint32_t IDESC_S = tc::idesc_bf16_f32(FW_BM, FW_BN, false, false);
    constexpr uint32_t IDESC_O = tc::idesc_bf16_f32(FW_BM, VC * 64, false, true);      // B = V is MN-major
    const uint64_t dQ = tc::smem_desc_kmajor_sw128(sQ);
    const uint64_t dK0 = tc::smem_desc_kmajor_sw128(sK(0));
    const uint64_t dV0 = tc::smem_desc_mnmajor_sw128(sV(0), FW_KV_CHUNK, 1024);
    auto issue_s = [&](int j) {
      const int sl = j & 1;
      tc::mbar_wait(k_full(sl), (j >> 1) & 1);
      tc::fence_after_sync();
      if (tc::elect_one()) {
        const uint64_t dK = dK0 + (uint64_t)sl * ((KC * FW_KV_CHUNK) >> 4);
        const uint32_t d = tS(j);
#pragma unroll
        for (int k = 0; k < 4 * KC; ++k)
          tc::mma_ss(d, dQ + (uint64_t)(((k >> 2) * FW_Q_CHUNK + (k & 3) * 32) >> 4),
                     dK + (uint64_t)(((k >> 2) * FW_KV_CHUNK + (k & 3) * 32) >> 4), IDESC_S, k != 0);
        tc::mma_commit(s_full(j & 1));
        tc::mma_commit(k_empty(sl));
      }
      __syncwarp();
    };
    tc::mbar_wait(q_full, 0);
    if (n_tiles > 0) issue_s(0);
    for (int j = 0; j < n_tiles; ++j) {
      if (j + 1 < n_tiles) issue_s(j + 1);               // S_{j+1} runs under softmax_j (its columns: P_{j-1}, whose P·V was issued before)
      const int sl = j & 1;
      tc::mbar_wait(v_full(sl), (j >> 1) & 1);
      tc::mbar_wait(p_full, j & 1);
      tc::fence_after_sync();
      if (tc::elect_one()) {
        const uint64_t dV = dV0 + (uint64_t)sl * ((VC * FW_KV_CHUNK) >> 4);
#pragma unroll
        for (int k = 0; k < FW_BN / 16; ++k) {
          tc::mma_ts(tO, tS(j) + k * 8, dV + (uint64_t)((k * 2048) >> 4), IDESC_O, j != 0 || k != 0);
          tc::mma_ts(tO, tS(j) + 32 + k * 8, dV + (uint64_t)((k * 2048) >> 4), IDESC_O, true);
        }
        tc::mma_commit(o_full);
        tc::mma_commit(v_empty(sl));
      }
      __syncwarp();
    }
  } else {
    const int quarter = warp & 3;                          // TMEM lane quadrant this warp may touch
    const int r = quarter * 32 + lane;                     // query row inside the tile
    const int slot = start + q0 + r;                       // cache slot (= causal limit) of this query
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const int lo_row = first_seen(slot), lo_warp = first_seen(start + q0 + quarter * 32 + 31);     // the largest bound of the warp
    const int lo_cta = first_seen(start + q0), hi_cta = start + q_hi;
    float m_ref = -INFINITY, l_run = 0.f;
    // rows [r0, r1) of a value tile (the swizzle moves 16-byte pieces within a row), the four warps together
    auto zero_rows = [&](uint32_t tile, int r0, int r1) {
      r0 = max(r0, 0);
      r1 = min(r1, FW_BN);
      for (int i = r0 * 8 + quarter * 32 + lane; i < r1 * 8; i += 128)
#pragma unroll
        for (int c = 0; c < VC; ++c)
          asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(tile + c * FW_KV_CHUNK + i * 16), "r"(0) : "memory");
    };

    for (int j = 0; j < n_tiles; ++j) {
      const int key0 = (first_tile + j) * FW_BN;
      const bool need_mask = (key0 + FW_BN - 1 > start + q0 + quarter * 32) || (key0 < lo_warp);     // warp-uniform
      tc::mbar_wait(s_full(j & 1), (j >> 1) & 1);
      tc::fence_after_sync();
      uint32_t v0[32], v1[32];
      tc::tmem_ld32(tS(j) + lane_off, v0);
      tc::tmem_ld32(tS(j) + lane_off + 32, v1);
      tc::tmem_ld_wait();
      if (need_mask) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (key0 + i > slot || key0 + i < lo_row) v0[i] = 0xff800000u;             // -inf
          if (key0 + 32 + i > slot || key0 + 32 + i < lo_row) v1[i] = 0xff800000u;
        }
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 32; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], fmaxf(__uint_as_float(v0[i]), __uint_as_float(v1[i])));
      const float t = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;
      const bool need = t > m_ref + FW_RESCALE || (m_ref == -INFINITY && t > -INFINITY);
      if (j == 0) {
        m_ref = t;
      } else if (__any_sync(0xffffffffu, need)) {
        const float factor = need ? exp2f(m_ref - t) : 1.0f;      // m_ref = -inf -> 0 (O and l are 0 there)
        tc::mbar_wait(o_full, (j - 1) & 1);                       // O at rest: P·V_{j-1} complete
        tc::fence_after_sync();
#pragma unroll 1
        for (int c = 0; c < 2 * VC; ++c) {
          uint32_t o[32];
          tc::tmem_ld32(tO + lane_off + c * 32, o);
          tc::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
          tc::tmem_st32(tO + lane_off + c * 32, o);
        }
        tc::tmem_st_wait();
        l_run *= factor;
        if (need) m_ref = t;
      }
      const float m_safe = m_ref == -INFINITY ? 0.f : m_ref;
      float psum0 = 0.f, psum1 = 0.f;
      auto split = [&](uint32_t (&v)[32], int at) {              // 32 scores -> packed pairs of hi at column `at`, of lo at 32 + at
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float a = fw_exp2(fmaf(__uint_as_float(v[2 * i]), p.scale_log2, -m_safe));
          const float c = fw_exp2(fmaf(__uint_as_float(v[2 * i + 1]), p.scale_log2, -m_safe));
          psum0 += a;
          psum1 += c;
          hi[i] = pack_bf16(a, c);
          lo[i] = pack_bf16(a - bf16_lo(hi[i]), c - bf16_hi(hi[i]));
        }
        tc::tmem_st16(tS(j) + lane_off + at, hi);
        tc::tmem_st16(tS(j) + lane_off + 32 + at, lo);
      };
      split(v0, 0);
      split(v1, 16);
      tc::tmem_st_wait();
      l_run += psum0 + psum1;
      if (key0 < lo_cta || key0 + FW_BN - 1 > hi_cta) {          // (uniform) the first or the last tile: slots that no query of the CTA sees
        tc::mbar_wait(v_full(j & 1), (j >> 1) & 1);
        zero_rows(sV(j & 1), 0, lo_cta - key0);
        zero_rows(sV(j & 1), hi_cta + 1 - key0, FW_BN);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");         // before the product that reads them
      }
      // at most one phase of p_full may be outstanding: P·V_{j-1} complete proves that the MMA warp consumed phase j-1 (flash_prefill.cu)
      if (j > 0) tc::mbar_wait(o_full, (j - 1) & 1);
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(p_full);
    }
    if (n_tiles > 0) {
      tc::mbar_wait(o_full, (n_tiles - 1) & 1);
      tc::fence_after_sync();
    }
    const bool row_on = q0 + r < p.S;
    const bool seen = !(l_run == 0.f);                       // (a sum that is NaN belongs to a query with a NaN or an infinite score: it stays NaN)
    float inv = 0.f;                                         // a query that sees nothing: its row is zero
    if (seen) inv = 1.0f / (l_run + (p.sink ? exp2f((p.sink_logit ? p.sink_logit[h] : 0.f) * 1.4426950408889634f - m_ref) : 0.f));
    if (p.gate != nullptr && row_on) inv *= sigmoid_f(p.gate[(size_t)(b * p.S + q0 + r) * p.ldg + h]);
    uint4* dst = reinterpret_cast<uint4*>(p.out + ((size_t)(b * p.S + q0 + r) * p.H + h) * (VC * 64));
#pragma unroll 1
    for (int c = 0; c < 2 * VC; ++c) {
      uint32_t o[32];
      if (n_tiles > 0) {
        tc::tmem_ld32(tO + lane_off + c * 32, o);
        tc::tmem_ld_wait();
      }
      if (!row_on) continue;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          w[e] = seen ? pack_bf16(__uint_as_float(o[8 * i + 2 * e]) * inv, __uint_as_float(o[8 * i + 2 * e + 1]) * inv) : 0u;
        dst[c * 4 + i] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    tc::fence_before_sync();
  }

  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 256);
}

template <int KC, int VC>
static int fw_launch(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FlashWide& p, cudaStream_t st) {
  const size_t smem = fw_smem_bytes(KC, VC);
  JL_CUDA(cudaFuncSetAttribute(flash_wide_kernel<KC, VC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  JL_CUDA(cudaFuncSetAttribute(flash_wide_kernel<KC, VC>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
  JL_CUDA(launch_pdl(flash_wide_kernel<KC, VC>, dim3((p.S + FW_BM - 1) / FW_BM, p.H, p.B), dim3(FW_THREADS), smem, st, tq, tk, tv, p));
  return JL_OK;
}

bool flash_wide_takes(int S, int D, int Dv, int T_cap, int ldk, int ldv, long long k_bs, long long k_hs, long long v_bs, long long v_hs,
                      const void* q, const void* k, const void* v, const void* out) {
  // TMA: 16-byte bases and strides; the tensor maps of a tile of 64 keys want a value row that is not shared with other channels
  auto stride_ok = [](long long s) { return s > 0 && s % 8 == 0; };
  return hybrid_tensor_cores() && S > 1 && T_cap >= 1 && D % 64 == 0 && D <= 256 && (Dv == 64 || Dv == 128) && ldk % 8 == 0 && ldv % 8 == 0 && stride_ok(k_bs) &&
         stride_ok(k_hs) && stride_ok(v_bs) && stride_ok(v_hs) && (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15) == 0;
}

int flash_wide_launch(const FlashWide& p, int D, int Dv, int T_cap, int ldk, int ldv, long long k_bs, long long k_hs, long long v_bs,
                      long long v_hs, const void* q, const void* k, const void* v, cudaStream_t st) {
  CUtensorMap tq, tk, tv;
  int rc = make_tmap_4d_bf16(&tq, q, D, p.S, p.H, p.B, (uint64_t)p.H * D, D, (uint64_t)p.S * p.H * D, FW_BM);
  if (rc) return rc;
  rc = make_tmap_4d_bf16(&tk, k, D, T_cap, p.G, p.B, ldk, k_hs, k_bs, FW_BN);
  if (rc) return rc;
  rc = make_tmap_4d_bf16(&tv, v, Dv, T_cap, p.G, p.B, ldv, v_hs, v_bs, FW_BN);
  if (rc) return rc;
  const int kc = D / 64;
  if (Dv == 128) {
    if (kc == 1) return fw_launch<1, 2>(tq, tk, tv, p, st);
    if (kc == 2) return fw_launch<2, 2>(tq, tk, tv, p, st);
    if (kc == 3) return fw_launch<3, 2>(tq, tk, tv, p, st);
    return fw_launch<4, 2>(tq, tk, tv, p, st);
  }
  if (kc == 1) return fw_launch<1, 1>(tq, tk, tv, p, st);
  if (kc == 2) return fw_launch<2, 1>(tq, tk, tv, p, st);
  if (kc == 3) return fw_launch<3, 1>(tq, tk, tv, p, st);
  return fw_launch<4, 1>(tq, tk, tv, p, st);
}

}  // namespace jl

// float32 linears of many rows on CTA pairs: the six bfloat16 products of linear_f32.cu, 256 features x BN rows per pair of SMs.
//
// A single CTA (linear_f32.cu) reads and cuts 128 + BN rows of 64 k for 128 x BN x 64 products, and the operands' way from the L2 bounds it
// long before the tensor core does.  Here the two CTAs of a pair each read and cut 128 features and HALF of the BN rows, and
// `tcgen05.mma.cta_group::2` multiplies all 256 features with all BN rows: twice the products for the same loads, cuts and shared
// memory.  The products of 64 k, their order and the rounded fp32 additions of their sums are those of the single CTA, so a sum over K that
// neither of them parts has the same bits.
//
//   * 8 producer warps per CTA read float32 rows, cut them into three bfloat16 parts each and write 2 x 3 swizzled tiles; both CTAs'
//     warps arrive on the leader's barrier;
//   * the leader's first epilogue warp issues 24 MMAs of 256 x BN x 16 per 64 k, the commit frees the stage in both CTAs;
//   * 8 epilogue warps per CTA add the finished sum (two in TMEM, alternating) to their registers: a thread owns one feature of BN / 2 rows.
// The (tile, 64 k) units of the whole product are dealt to the pairs in even runs, so that no round of tiles is incomplete: a run that ends
// inside a tile leaves a partial tile in the workspace, and a second kernel adds a tile's parts in order of k.  Where whole tiles are as fast
// there is no second kernel.  A long chain of additions costs precision: what is more than LP_FOLD units, or than a CTA of linear_f32.cu adds in a row for the same product, is
// folded through the workspace on its way.
// Bound: 24 MMAs of 12 BN cycles together per unit, with the loads (64 KB per CTA and unit at BN 256) and the folds right behind: tensor pipe 59 % active, load and store pipe 53 %
// (200 x 10928 x 2048).  One B200, single CTAs -> this, us (rows x features x K): 200 x 10928 x 2048 153 -> 58 (52 with sums of 32 units), 200 x 2048 x 5464 54 -> 35, 128 x 10928 x 2048 78 -> 43, 1000 x 1024 x 1024 31.5 -> 22, 2048 x 6176 x 1024
// 263 -> 128, 2048 x 10928 x 2048 759 -> 400.  Error against float64 (2-norm), normal operands; one sign: 200 x 10928 x 2048 1.04e-7 -> 1.05e-7 (1.13e-7 with sums of 32); 9.6e-8 -> 9.7e-8,
// 200 x 2048 x 5464 1.25e-7 -> 1.16e-7; 9.6e-8 -> 9.8e-8, 2048 x 6176 x 1024 1.09e-7 -> 1.07e-7; 1.07e-7 -> 1.04e-7, 2048 x 10928 x 2048 1.31e-7 -> 1.29e-7; 1.23e-7 -> 1.20e-7,
// 400 x 512 x 512 9.2e-8 -> 9.1e-8; 9.5e-8 -> 9.4e-8.  (Sums are added as they come: a factor on them against the mean of what the tensor core cuts off would change those that are exact.)
#include "jllama_b200.h"
#include "linear_f32.cuh"
#include "seq_types.cuh"
#include "tcgen05.cuh"

namespace jl {

constexpr int LP_BM = 128, LP_BK = 64, LP_PROD = 8, LP_EPI = 8, LP_THREADS = (LP_PROD + LP_EPI) * 32;
constexpr uint32_t LP_A_BYTES = LP_BM * LP_BK * 2;                   // one part of a CTA's weights
constexpr int LP_STAGES = 2, LP_FOLD = 32;
constexpr uint32_t lp_stage_bytes(int bn) { return 3 * (LP_A_BYTES + bn / 2 * LP_BK * 2); }
constexpr size_t lp_smem(int bn) { return LP_STAGES * lp_stage_bytes(bn) + 1024; }
constexpr int LP_PROD_REGS = 104, LP_EPI_REGS = 152;                 // 256 threads each: together the 128 x 512 of the launch

struct LinearPair {
  const float* x; const float* w; float* out; float* ws;
  int ldx, ldo, M, N, K;
  int m_tiles, tiles, blocks, pairs, split;                          // blocks: of 64 k per tile; split: runs may end inside a tile
  int fold;                                                          // most units that are added in a row
  int slots;                                                         // partial tiles that a pair keeps in the workspace
};

// first unit of a pair's run
__host__ __device__ __forceinline__ long long lp_begin(const LinearPair& p, int pair) {
  return p.split ? (long long)p.tiles * p.blocks * pair / p.pairs : (long long)p.blocks * ((long long)p.tiles * pair / p.pairs);
}
// Floats of a partial tile.  Where runs end inside tiles a pair leaves at most two (slot 0 continues a tile, slot 1 begins one); where a run has more units of a tile than are
// added in a row, the sum so far lies in its last slot.
__host__ __device__ __forceinline__ size_t lp_part(int bn) { return (size_t)2 * LP_BM * bn; }

__device__ __forceinline__ void lp_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)acc)
      : "memory");
}
__device__ __forceinline__ void lp_commit_both(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ uint32_t lp_leader(uint32_t addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void lp_arrive(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void lp_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// the same sum with FMAs in order of k, for an output that is not finite
__device__ __forceinline__ float lp_again(const float* xr, const float* wr, int K) {
  float s = 0.0f;
#pragma unroll 1
  for (int k = 0; k < K; ++k) s = fmaf(xr[k], wr[k], s);
  return s;
}

template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(LP_THREADS, 1) linear_f32_pair_kernel(const LinearPair p) {
  constexpr int HALF = BN / 2, STEP = LP_PROD * 4, NW = LP_BM / STEP, NX = (HALF + STEP - 1) / STEP;
  constexpr uint32_t STAGE = lp_stage_bytes(BN), B_BYTES = HALF * LP_BK * 2, B_OFF = 3 * LP_A_BYTES;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(8) unsigned long long bar_mem[2 * LP_STAGES + 4];
  __shared__ uint32_t tmem_slot;
  const uint32_t raw = tc::smem_u32(smem_raw), base = (raw + 1023u) & ~1023u, bars = tc::smem_u32(bar_mem);
  auto full = [&](int s) { return bars + 8u * s; };
  auto empty = [&](int s) { return bars + 8u * (LP_STAGES + s); };
  auto tfull = [&](int s) { return bars + 8u * (2 * LP_STAGES + s); };
  auto tempty = [&](int s) { return bars + 8u * (2 * LP_STAGES + 2 + s); };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1;

  if (warp == LP_PROD) {                                             // the same warp of both CTAs
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(&tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    if (lane == 0) {
      for (int s = 0; s < LP_STAGES; ++s) { tc::mbar_init(full(s), 2 * LP_PROD); tc::mbar_init(empty(s), 1); }
      for (int s = 0; s < 2; ++s) { tc::mbar_init(tfull(s), 1); tc::mbar_init(tempty(s), 2 * LP_EPI); }
      tc::fence_barrier_init();
    }
  }
  tc::fence_before_sync();
  lp_cluster_sync();                                                 // barriers of both CTAs exist before any arrival from the other
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  pdl_wait();
  pdl_launch_dependents();
  const long long first = lp_begin(p, pair);
  const int n = (int)(lp_begin(p, pair + 1) - first);                // units of this run
  const int tile0 = (int)(first / p.blocks), kb0 = (int)(first % p.blocks);

  if (warp < LP_PROD) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(LP_PROD_REGS));
    const int r = threadIdx.x / 8, c = threadIdx.x & 7;              // 8 lanes take the 64 k of a row, 8 each
    uint32_t src[NW + NX];                                           // (the host checks that both operands have fewer than 2^31 elements)
    auto set_tile = [&](int t) {
      const int n0 = t / p.m_tiles * (2 * LP_BM) + rank * LP_BM, m0 = t % p.m_tiles * BN + rank * HALF;
      // rows beyond the matrix repeat its last one: their outputs are not stored
#pragma unroll
      for (int i = 0; i < NW; ++i) src[i] = (uint32_t)min(n0 + r + i * STEP, p.N - 1) * (uint32_t)p.K + 8 * c;
#pragma unroll
      for (int i = 0; i < NX; ++i) src[NW + i] = (uint32_t)min(m0 + r + i * STEP, p.M - 1) * (uint32_t)p.ldx + 8 * c;
    };
    float4 va[NW + NX], vb[NW + NX];                                 // the next block of 64 k
    auto on = [&](int i) { return i < NW + HALF / STEP || HALF % STEP == 0 || r < HALF % STEP; };     // (uniform for a warp)
    uint32_t at = 0;
    bool ina = true, inb = true;                                     // the last block: K is a multiple of four
    auto set_block = [&](int kb) {
      at = (uint32_t)kb * LP_BK;
      ina = (int)at + 8 * c < p.K;
      inb = (int)at + 8 * c + 4 < p.K;
    };
    auto load = [&](int i) {
      const float* s = (i < NW ? p.w : p.x) + (src[i] + at);
      va[i] = ina ? *reinterpret_cast<const float4*>(s) : make_float4(0.f, 0.f, 0.f, 0.f);
      vb[i] = inb ? *reinterpret_cast<const float4*>(s + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    const uint32_t lane_off = base + r * 128 + ((c ^ (r & 7)) << 4);         // (STEP rows further: the same swizzle)
    const uint32_t full0 = lp_leader(full(0));
    int tile = tile0, kb = kb0;
    if (n > 0) {
      set_tile(tile);
      set_block(kb);
#pragma unroll
      for (int i = 0; i < NW + NX; ++i) if (on(i)) load(i);
    }
#pragma unroll 1
    for (int u = 0; u < n; ++u) {
      const int stage = u % LP_STAGES;
      const bool more = u + 1 < n;
      if (more) {
        if (++kb == p.blocks) { kb = 0; set_tile(++tile); }
        set_block(kb);
      }
      tc::mbar_wait(empty(stage), ((u / LP_STAGES) & 1) ^ 1);
      const uint32_t st = lane_off + stage * STAGE;
#pragma unroll
      for (int i = 0; i < NW + NX; ++i) {
        if (!on(i)) continue;
        uint4 h[3];
        lf_split8(va[i], vb[i], h);
        const uint32_t dst = st + (i < NW ? i * STEP * 128 : B_OFF + (i - NW) * STEP * 128);
#pragma unroll
        for (int k = 0; k < 3; ++k)
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + k * (i < NW ? LP_A_BYTES : B_BYTES)), "r"(h[k].x), "r"(h[k].y),
                       "r"(h[k].z), "r"(h[k].w) : "memory");
        if (more) load(i);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // these writes -> visible to the tensor core
      __syncwarp();
      if (lane == 0) lp_arrive(full0 + 8u * stage);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(LP_EPI_REGS));
    constexpr uint32_t IDESC = tc::idesc_bf16_f32(2 * LP_BM, BN);
    // the leader's first epilogue warp also issues: the MMAs of the next unit go out before it waits for the current sum
    auto issue = [&](int u) {
      const int buf = u & 1, stage = u % LP_STAGES;
      tc::mbar_wait(tempty(buf), ((u >> 1) & 1) ^ 1);
      tc::mbar_wait(full(stage), (u / LP_STAGES) & 1);
      tc::fence_after_sync();
      if (tc::elect_one()) {
        const uint64_t da0 = tc::smem_desc_kmajor_sw128(base + stage * STAGE), db0 = da0 + (B_OFF >> 4);
        const uint32_t d = tmem + buf * 256;
        // parts of the weights and of the rows, the smallest products first
        constexpr int PA[6] = {0, 2, 1, 0, 1, 0}, PB[6] = {2, 0, 1, 1, 0, 0};
#pragma unroll
        for (int q = 0; q < 6; ++q) {
#pragma unroll
          for (int k = 0; k < LP_BK / 16; ++k)
            lp_mma(d, da0 + ((PA[q] * LP_A_BYTES >> 4) + 2 * k), db0 + ((PB[q] * B_BYTES >> 4) + 2 * k), IDESC, q != 0 || k != 0);
        }
        lp_commit_both(empty(stage));
        lp_commit_both(tfull(buf));
      }
      __syncwarp();
    };
    const bool issuer = rank == 0 && warp == LP_PROD;
    const int half = (warp - LP_PROD) >> 2, feature = (warp & 3) * 32 + lane;
    const uint32_t row = tmem + ((uint32_t)((warp & 3) * 32) << 16) + half * HALF;
    const uint32_t tempty0 = lp_leader(tempty(0));
    if (issuer && n > 0) issue(0);
    int tile = tile0, kb = kb0;
#pragma unroll 1
    for (int u = 0; u < n; ++tile, kb = 0) {                         // the tiles of this run
      const int kstart = kb, units = min(p.blocks - kb, n - u);
      float* const sofar = p.ws + ((size_t)(pair + 1) * p.slots - 1) * lp_part(BN) + (size_t)half * HALF * (2 * LP_BM) + rank * LP_BM + feature;
      float acc[HALF];
#pragma unroll 1
      for (int done = 0; done < units; done += p.fold) {             // sums of `fold` units, which then meet
#pragma unroll
        for (int j = 0; j < HALF; ++j) acc[j] = 0.0f;
#pragma unroll 1
        for (const int end = u + min(p.fold, units - done); u < end; ++u) {
          const int buf = u & 1;
          if (issuer && u + 1 < n) issue(u + 1);
          tc::mbar_wait(tfull(buf), (u >> 1) & 1);
          tc::fence_after_sync();
#pragma unroll
          for (int c0 = 0; c0 < HALF; c0 += 16) {
            uint32_t v[16];
            tc::tmem_ld16(row + buf * 256 + c0, v);
            tc::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[c0 + j] += __uint_as_float(v[j]);
          }
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) lp_arrive(tempty0 + 8u * buf);
        }
        if (done > 0) {
#pragma unroll
          for (int j = 0; j < HALF; ++j) acc[j] += sofar[(size_t)j * (2 * LP_BM)];
        }
        if (done + p.fold < units) {
#pragma unroll
          for (int j = 0; j < HALF; ++j) sofar[(size_t)j * (2 * LP_BM)] = acc[j];
        }
      }
      if (units < p.blocks) {                                        // a part of the tile
        float* o = p.ws + ((size_t)pair * p.slots + (kstart == 0)) * lp_part(BN) + (size_t)half * HALF * (2 * LP_BM) + rank * LP_BM + feature;
#pragma unroll
        for (int j = 0; j < HALF; ++j) o[(size_t)j * (2 * LP_BM)] = acc[j];
      } else {
        const int nf = tile / p.m_tiles * (2 * LP_BM) + rank * LP_BM + feature, m0 = tile % p.m_tiles * BN + half * HALF, rows = nf < p.N ? min(HALF, p.M - m0) : 0;
        float* const o = p.out + (size_t)m0 * p.ldo + nf;
        float* to = o;
        bool bad = false;
#pragma unroll
        for (int j = 0; j < HALF; ++j) {
          if (j < rows) {
            *to = acc[j];
            bad |= !(fabsf(acc[j]) < INFINITY);
          }
          to += p.ldo;
        }
        if (bad)
          for (int j = 0; j < rows; ++j)
            if (!(fabsf(o[(size_t)j * p.ldo]) < INFINITY))
              o[(size_t)j * p.ldo] = lp_again(p.x + (size_t)(m0 + j) * p.ldx, p.w + (size_t)nf * p.K, p.K);
      }
      __syncwarp();                                                  // lanes whose feature or rows lie outside have not waited
    }
  }
  tc::fence_before_sync();
  lp_cluster_sync();                                                 // neither CTA frees its tensor memory while the pair still uses it
  if (warp == LP_PROD) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// The tiles that several pairs took parts of: their sums, in order of k.  grid (tiles, BN / 16 groups of rows), a thread takes four features of four rows.
constexpr int LPS_ROWS = 16, LPS_THREADS = 256;

__global__ void __launch_bounds__(LPS_THREADS) linear_f32_pair_sum_kernel(const LinearPair p, int bn) {
  pdl_wait();
  pdl_launch_dependents();
  const int tile = blockIdx.x;
  const long long total = (long long)p.tiles * p.blocks, u0 = (long long)tile * p.blocks, u1 = u0 + p.blocks - 1;
  const int p0 = (int)(((u0 + 1) * p.pairs - 1) / total), p1 = (int)(((u1 + 1) * p.pairs - 1) / total);      // owners of its first and last unit
  if (p0 == p1) return;                                              // written by one pair
  const int c = (threadIdx.x & 63) * 4, r0 = blockIdx.y * LPS_ROWS + (threadIdx.x >> 6);
  const int nf = tile / p.m_tiles * (2 * LP_BM) + c, m0 = tile % p.m_tiles * bn;
  const size_t part = lp_part(bn);
  const float* src = p.ws + (size_t)r0 * (2 * LP_BM) + c;
  float4 s[LPS_ROWS / 4];
#pragma unroll
  for (int i = 0; i < LPS_ROWS / 4; ++i) s[i] = *reinterpret_cast<const float4*>(src + ((size_t)p0 * p.slots + 1) * part + (size_t)i * 4 * (2 * LP_BM));
  for (int q = p0 + 1; q <= p1; ++q) {
    float4 v[LPS_ROWS / 4];
#pragma unroll
    for (int i = 0; i < LPS_ROWS / 4; ++i) v[i] = *reinterpret_cast<const float4*>(src + (size_t)q * p.slots * part + (size_t)i * 4 * (2 * LP_BM));
#pragma unroll
    for (int i = 0; i < LPS_ROWS / 4; ++i) { s[i].x += v[i].x; s[i].y += v[i].y; s[i].z += v[i].z; s[i].w += v[i].w; }
  }
  const bool wide = ((uintptr_t)p.out & 15) == 0 && p.ldo % 4 == 0;
#pragma unroll
  for (int i = 0; i < LPS_ROWS / 4; ++i) {
    const int m = m0 + r0 + i * 4;
    if (r0 + i * 4 >= bn || m >= p.M) continue;
    float v[4] = {s[i].x, s[i].y, s[i].z, s[i].w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (nf + j < p.N && !(fabsf(v[j]) < INFINITY)) v[j] = lp_again(p.x + (size_t)m * p.ldx, p.w + (size_t)(nf + j) * p.K, p.K);
    float* o = p.out + (size_t)m * p.ldo + nf;
    if (wide && nf + 4 <= p.N) *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
    else
      for (int j = 0; j < 4; ++j) if (nf + j < p.N) o[j] = v[j];
  }
}

// Rows per tile, and whether runs end inside tiles: the least time in us, from what the busiest pair takes to begin, per unit, tile and fold, and what partial tiles
// cost (fitted to 130 sizes with every choice of the two and weights out of memory: 6 % off in the mean, its picks 0.3 % above the best).  False: the single CTAs are faster.
static bool lp_plan(int M, int N, int K, int num_sms, LinearPair& p, int& bn) {
  static const struct { int bn; double unit; } shapes[] = {{256, 2.47}, {224, 2.11}, {192, 1.77}, {128, 1.28}};
  const LinearF32Plan single = linear_f32_plan(M, N, K);
  double best = 1e300;
  p.fold = single.chain < LP_FOLD ? single.chain : LP_FOLD;
  for (const auto& sh : shapes) {
    const int mt = (M + sh.bn - 1) / sh.bn, tiles = mt * ((N + 2 * LP_BM - 1) / (2 * LP_BM)), blocks = (K + LP_BK - 1) / LP_BK;
    for (int split = 0; split < 2; ++split) {
      int pairs = num_sms / 2;
      if (!split && pairs > tiles) pairs = tiles;
      if (split && (long long)pairs * 4 > (long long)tiles * blocks) pairs = tiles * blocks / 4;
      if (pairs < 1) continue;
      const long long units = split ? ((long long)tiles * blocks + pairs - 1) / pairs : (long long)((tiles + pairs - 1) / pairs) * blocks;
      const int run = units < blocks ? (int)units : blocks;                 // most units of a tile
      const double of_run = (double)units / run;
      const double t = 3.9 + sh.unit * units + of_run * (1.6 + 2.4 * ((run - 1) / p.fold) * sh.bn / 256) +
                       (split ? 0.4 + (double)blocks / run * (0.26 + 0.48e-3 * (tiles < pairs ? tiles : pairs) * sh.bn) : 0.0);
      if (t < (sh.bn == bn ? best : 0.97 * best)) {                         // (fewer rows a tile: more ways of the weights through the L2)
        best = t; bn = sh.bn;
        p.m_tiles = mt; p.tiles = tiles; p.blocks = blocks; p.pairs = pairs; p.split = split;
        p.slots = (split ? 2 : 0) + (run > p.fold);
      }
    }
  }
  // What the single CTAs take, likewise, with as many clusters of 2, 4 and 8 at once as find a place.  Of 1806 sizes (65 to 2500 rows, 256 to 12000 features, K 256 to 8200, weights out
  // of memory) six that go to the pairs are slower there by more than 2 % (at most 11 %), 64 that stay would be faster by more than 3 % (at most 18 %).  Near the line, us, single CTAs |
  // pairs: 300 x 300 x 512 8.1 | 12.8, 512 x 256 x 1024 10.2 | 12.0, 128 x 2048 x 1024 13.1 | 13.7, 160 x 512 x 2048 13.8 | 16.2, 288 x 908 x 356 10.5 | 14.0; 257 x 256 x 256 9.7 | 9.0,
  // 540 x 674 x 884 18.8 | 15.9, 257 x 256 x 4096 26.9 | 16.1.
  const int at_once = single.splits == 8 ? 15 : single.splits == 4 ? 33 : num_sms / single.splits;
  const double more = single.splits == 8 ? -1.9 : single.splits == 4 ? -0.8 : single.splits == 2 ? 1.9 : 0.0, block = single.bn == 32 ? 0.80 : single.bn == 64 ? 1.36 : 2.43;
  return best < 1.1 + (double)((single.tiles + at_once - 1) / at_once) * (7.0 + more + block * single.chain);
}

template <int BN>
static cudaError_t lp_launch(const LinearPair& p, cudaStream_t st) {
  auto* kernel = linear_f32_pair_kernel<BN>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lp_smem(BN));
  if (e != cudaSuccess) return e;
  return launch_pdl(kernel, dim3(2 * p.pairs), dim3(LP_THREADS), lp_smem(BN), st, p);
}

}  // namespace jl

using namespace jl;

// Where it may beat the single CTAs (lp_plan compares; us, single CTAs | this: 128 x 1024 x 1024 10.4 | 11.9, 256 x 512 x 1024 10.4 | 12.2, 256 x 1024 x 512 10.2 | 11.3); 16-byte
// loads along K.
static bool lp_takes(int M, int N, int K, int ldx, const void* x, const void* w) {
  return M > 64 && N >= 256 && (M > 256 || (long long)N * K >= (M > 128 ? 1 << 20 : 1 << 21)) && K >= 256 && K % 4 == 0 && ldx % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0 && (long long)N * K < (1ll << 31) &&
         (long long)M * ldx < (1ll << 31);
}

extern "C" JL_API long long jl_linear_f32_pair_ws(const void* x, int ldx, const void* w, int M, int N, int K, int num_sms) {
  if (!lp_takes(M, N, K, ldx, x, w)) return -1;
  LinearPair p{};
  int bn = 0;
  if (!lp_plan(M, N, K, num_sms, p, bn)) return -1;
  return (long long)((size_t)p.pairs * p.slots * lp_part(bn) * sizeof(float));
}

extern "C" JL_API int jl_linear_f32_pair(const void* x, int ldx, const void* w, void* out, int ldo, int M, int N, int K, int num_sms, void* ws,
                                         void* stream) {
  if (!lp_takes(M, N, K, ldx, x, w)) return JL_ERR_UNSUPPORTED;
  JL_CHECK_ARG(ldx >= K && ldo >= N, "jl_linear_f32_pair: bad pitch ldx=%d ldo=%d (N=%d K=%d)", ldx, ldo, N, K);
  LinearPair p{};
  int bn = 0;
  if (!lp_plan(M, N, K, num_sms, p, bn)) return JL_ERR_UNSUPPORTED;
  JL_CHECK_ARG(p.slots == 0 || (ws != nullptr && ((uintptr_t)ws & 15) == 0), "jl_linear_f32_pair: a workspace of 16-byte alignment is needed");
  p.x = (const float*)x; p.w = (const float*)w; p.out = (float*)out; p.ws = (float*)ws;
  p.ldx = ldx; p.ldo = ldo; p.M = M; p.N = N; p.K = K;
  cudaStream_t st = (cudaStream_t)stream;
  JL_CUDA(bn == 128 ? lp_launch<128>(p, st) : bn == 192 ? lp_launch<192>(p, st) : bn == 224 ? lp_launch<224>(p, st) : lp_launch<256>(p, st));
  if (p.split) JL_CUDA(launch_pdl(linear_f32_pair_sum_kernel, dim3(p.tiles, bn / LPS_ROWS), dim3(LPS_THREADS), 0, st, p, bn));
  return JL_OK;
}

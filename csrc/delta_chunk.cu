// Gated delta rule with one decay per head over a prompt, 32 tokens at a time, in fp32 FMAs.
//
// With unit keys k_i, queries q_i (times D^(-1/2)), decays a_i, A_i = a_1 ... a_i and r_ij = a_(j+1) ... a_i, the tokens of a chunk that starts
// from the state S obey  e_i = beta_i (v_i - A_i k_i.S - sum_{j<i} r_ij k_i.k_j e_j),  o_i = A_i q_i.S + sum_{j<=i} r_ij q_i.k_j e_j.
// The sum over earlier tokens is a unit lower triangular system, I + M with M_ij = beta_i r_ij k_i.k_j (the WY form of a product of Householder-like
// factors; Yang, Wang, Zhang, Shen, Kim, "Parallelizing Linear Transformers with the Delta Rule over Sequence Length", 2024).  So
//     E = T (V - (A K) S) with T = (I + M)^-1 diag(beta),   O = (A Q) S + P E with P_ij = r_ij q_i.k_j,   S <- A_32 S + (r_32 K)^T E.
// Products of decays are running products, never quotients: a decay of zero is an ordinary value.
//
// delta_chunk_prep_kernel forms A K | A Q | (r_32 K)^T | T | P | A_32 of every chunk and head, all chunks at once; delta_chunk_scan_kernel walks the
// chunks of its head and slice of value columns: the record of the next chunk comes by one bulk copy meanwhile.  All products are dot
// products along contiguous numbers: four rows x TC columns per thread, two FMAs an instruction (fma.rn.f32x2), the state in registers and, for the next
// chunk's dot products, in shared memory by columns.
// Bound: FMA issue of the few warps that the heads and columns give (64 x 128 keys x values, 32 tokens: 960 packed FMAs a thread, and three barriers).
// Shared memory is what the walk asks most of (61 % of its wavefronts, 44 % of the FMA
// pipe, 39 % of the issue slots).  One B200, 2 rows x 1000 tokens x 16 heads of 64 x 128, blocks of four tokens one after the other -> this: both launches 350 -> 101 us, the
// layer 383 -> 217; 4 x 512 x 16 heads of 128 x 128 298 -> 188, 1 x 2048 x 4 heads of 128 x 128 481 -> 145, 1 x 24 x 4 heads of 32 x 64 12.4 -> 12.5, 8 x 2000 x 16 heads of
// 64 x 128 1125 -> 695.  Error against float64 (2-norm of the read-outs, of the state): 2.0e-7, 2.0e-7 -> 1.9e-7, 1.9e-7; 128 channels 2.1e-7, 3.0e-7 -> 2.1e-7, 2.9e-7.
#include "delta_chunk.cuh"
#include "jllama_b200.h"
#include "seq_types.cuh"
#include "tcgen05.cuh"

namespace jl {

constexpr int DC_CTAS = 200;
constexpr int DC_T = 32, DC_THREADS = 128, DC_TP = DC_T + 4;         // tokens of a chunk; threads; pitch of a row of 32 (rows on distinct banks)
// record of a chunk and head: A K rows | A Q rows (pitch D + 4) | (r K)^T rows, T rows, P rows (pitch 36) | A_32, three unused
template <int D> struct DcRecord {
  static constexpr int KP = D + 4, Q = DC_T * KP, KT = 2 * DC_T * KP, T = KT + D * DC_TP, P = T + DC_T * DC_TP, A = P + DC_T * DC_TP, FLOATS = A + 4;
};
static size_t dc_record_floats(int D) { return D <= 32 ? DcRecord<32>::FLOATS : D <= 64 ? DcRecord<64>::FLOATS : DcRecord<128>::FLOATS; }

__device__ __forceinline__ unsigned long long dc_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long dc_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long dc_add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float dc_sum2(unsigned long long a) { return __uint_as_float((uint32_t)a) + __uint_as_float((uint32_t)(a >> 32)); }

// acc[i][j] += rows[i] . cols[j] over N numbers (a multiple of four, 16-byte aligned); two partial sums each, and sums of 16 numbers before they
// join the longer ones
template <int R, int C, int N>
__device__ __forceinline__ void dc_dot(unsigned long long (&acc)[R][C], const float* const (&row)[R], const float* const (&col)[C]) {
#pragma unroll 2
  for (int k0 = 0; k0 < N; k0 += 16) {
    unsigned long long part[R][C];
#pragma unroll
    for (int k = k0; k < k0 + 16; k += 4) {
      ulonglong2 a[R], b[C];
#pragma unroll
      for (int i = 0; i < R; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(row[i] + k);
#pragma unroll
      for (int j = 0; j < C; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(col[j] + k);
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) part[i][j] = dc_fma2(a[i].y, b[j].y, k == k0 ? dc_mul2(a[i].x, b[j].x) : dc_fma2(a[i].x, b[j].x, part[i][j]));
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < C; ++j) acc[i][j] = dc_add2(acc[i][j], part[i][j]);
  }
}

// Of the 16 x 8 rows and columns of a CTA's tile a thread's first ones; a warp has four rows x eight columns.  Which lanes share a row decides what a
// 16-byte shared-memory load costs: rows by lane bits 0 and 2 take 113 us where rows by lane / 8 take 127 (the case below).
__device__ __forceinline__ int dc_row(int tid) { return (tid >> 5) * 4 + (tid & 1) + ((tid >> 2) & 1) * 2; }
__device__ __forceinline__ int dc_col(int tid) { return ((tid >> 1) & 1) + ((tid >> 3) & 3) * 2; }

__device__ __forceinline__ int dc_first(const DeltaHeadParams& p, int b) { return max(0, (p.pad_left ? p.pad_left[b] : 0) - (p.cache_len ? *p.cache_len : 0)); }

// grid (chunks, heads, rows), 128 threads.  D: channels of a key, padded with zeros to 32, 64 or 128.
template <typename T, int D>
__global__ void __launch_bounds__(DC_THREADS, D <= 64 ? 7 : 4) delta_chunk_prep_kernel(DeltaHeadParams p, float* ws, const T* __restrict__ a_bias,
                                                                      const T* __restrict__ a_log) {
  pdl_wait();                      // programmatic dependent launch: nothing is read before the predecessor is done
  pdl_launch_dependents();
  using R = DcRecord<D>;
  extern __shared__ float4 smem4[];
  float* ks = reinterpret_cast<float*>(smem4);                 // unit keys, rows of KP | queries
  float* qs = ks + DC_T * R::KP;
  float* ratio = qs + DC_T * R::KP;                            // [i][j], pitch 33
  float* ms = ratio + DC_T * 33;                               // M, pitch 36
  float* as = ms + DC_T * DC_TP;                               // A_i | a_i | beta_i
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y, b = blockIdx.z, g = h / (p.H / p.G);
  const int s0 = dc_first(p, b) + (int)blockIdx.x * DC_T, nt = min(DC_T, p.S - s0);
  if (nt <= 0) return;
  const size_t m0 = (size_t)b * p.S + s0;
  float* rec = ws + (((size_t)b * p.H + h) * gridDim.x + blockIdx.x) * R::FLOATS;
  {                                                            // eight tokens per warp, all loads first: unit keys, queries times D^(-1/2)
    constexpr int NT = DC_T * 32 / DC_THREADS;
    float kv[NT][D / 32], qv[NT][D / 32];
#pragma unroll
    for (int x = 0; x < NT; ++x) {
      const int i = warp * NT + x;
      const float* ur = p.u + (m0 + i) * p.ldu + g * p.D;
#pragma unroll
      for (int r = 0; r < D / 32; ++r) {
        const int d = r * 32 + lane;
        const bool in = i < nt && d < p.D;
        kv[x][r] = in ? ur[p.k_off + d] : 0.0f;
        qv[x][r] = in ? ur[p.q_off + d] : 0.0f;
      }
    }
#pragma unroll
    for (int x = 0; x < NT; ++x) {
      float kk = 0.0f, qq = 0.0f;
#pragma unroll
      for (int r = 0; r < D / 32; ++r) { kk = fmaf(kv[x][r], kv[x][r], kk); qq = fmaf(qv[x][r], qv[x][r], qq); }
      kk = warp_sum(kk); qq = warp_sum(qq);
      const float rq = 1.0f / sqrtf(qq + 1e-6f) / sqrtf((float)p.D), rk = 1.0f / sqrtf(kk + 1e-6f);
#pragma unroll
      for (int r = 0; r < D / 32; ++r) {
        ks[(warp * NT + x) * R::KP + r * 32 + lane] = kv[x][r] * rk;
        qs[(warp * NT + x) * R::KP + r * 32 + lane] = qv[x][r] * rq;
      }
    }
  }
  if (tid < DC_T) {                                            // tokens beyond the row: no decay, no correction
    const bool in = tid < nt;
    const float* yr = p.y + (m0 + tid) * p.ldy;
    as[DC_T + tid] = in ? delta_head_decay(yr[p.a_off + h] + to_f(a_bias[h]), to_f(a_log[h])) : 1.0f;
    as[2 * DC_T + tid] = in ? sigmoid_f(yr[p.b_off + h]) : 0.0f;
  }
  __syncthreads();
  if (warp == 0) {                                             // lane j: r_ij for i >= j
    float r = 1.0f;
#pragma unroll
    for (int i = 0; i < DC_T; ++i) {
      if (i > lane) r *= as[DC_T + i];
      ratio[i * 33 + lane] = i < lane ? 0.0f : r;
    }
  } else if (tid == 32) {
    float r = 1.0f;
    for (int i = 0; i < DC_T; ++i) { r *= as[DC_T + i]; as[i] = r; }
    rec[R::A] = r; rec[R::A + 1] = 0.0f; rec[R::A + 2] = 0.0f; rec[R::A + 3] = 0.0f;
  }
  __syncthreads();
  const int rg = dc_row(tid), cg = dc_col(tid);                // rows rg, rg + 16 of K and of Q x tokens cg + 8 j
  {
    unsigned long long acc[4][4] = {};
    const float* row[4] = {ks + rg * R::KP, ks + (rg + 16) * R::KP, qs + rg * R::KP, qs + (rg + 16) * R::KP};
    const float* col[4] = {ks + cg * R::KP, ks + (cg + 8) * R::KP, ks + (cg + 16) * R::KP, ks + (cg + 24) * R::KP};
    dc_dot<4, 4, D>(acc, row, col);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = rg + 16 * i, c = cg + 8 * j;
        ms[r * DC_TP + c] = c < r ? as[2 * DC_T + r] * (ratio[r * 33 + c] * dc_sum2(acc[i][j])) : 0.0f;
        rec[R::P + r * DC_TP + c] = c <= r ? ratio[r * 33 + c] * dc_sum2(acc[2 + i][j]) : 0.0f;
      }
  }
  __syncthreads();
  if (warp == 0) {                                             // (I + M)^-1, a column per lane
    float t[DC_T];
#pragma unroll
    for (int i = 0; i < DC_T; ++i) {
      float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int m = 0; m < i; m += 4) {
        const float4 v = *reinterpret_cast<const float4*>(ms + i * DC_TP + m);
        s[0] = m >= lane ? fmaf(v.x, t[m], s[0]) : s[0];       // (t[m] = 0 for m < lane; nothing that is not finite may come from there)
        if (m + 1 < i) s[1] = m + 1 >= lane ? fmaf(v.y, t[m + 1], s[1]) : s[1];
        if (m + 2 < i) s[2] = m + 2 >= lane ? fmaf(v.z, t[m + 2], s[2]) : s[2];
        if (m + 3 < i) s[3] = m + 3 >= lane ? fmaf(v.w, t[m + 3], s[3]) : s[3];
      }
      t[i] = i < lane ? 0.0f : i == lane ? 1.0f : -((s[0] + s[1]) + (s[2] + s[3]));
      rec[R::T + i * DC_TP + lane] = i < lane ? 0.0f : t[i] * as[2 * DC_T + lane];
    }
  } else {
    for (int x = tid - 32; x < DC_T * D; x += DC_THREADS - 32) {
      const int i = x / D, d = x % D;
      rec[i * R::KP + d] = as[i] * ks[i * R::KP + d];
      rec[R::Q + i * R::KP + d] = as[i] * qs[i * R::KP + d];
    }
    for (int x = tid - 32; x < DC_T * D; x += DC_THREADS - 32) {
      const int d = x / DC_T, m = x % DC_T;
      rec[R::KT + d * DC_TP + m] = ratio[(DC_T - 1) * 33 + m] * ks[m * R::KP + d];
    }
  }
}

__device__ __forceinline__ void dc_cp16(float* dst, const float* src, bool on) {          // 16 bytes, zeros where there is nothing to copy
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");
}

// grid (slices of 8 TC value columns, heads, rows), 128 threads
template <int D, int TC>
__global__ void __launch_bounds__(DC_THREADS) delta_chunk_scan_kernel(DeltaHeadParams p, const float* ws, int chunks, int wide) {
  pdl_wait();                      // programmatic dependent launch: nothing is read before the predecessor is done
  pdl_launch_dependents();
  using R = DcRecord<D>;
  constexpr int COLS = 8 * TC, VP = COLS + 8, DR = D / 16;      // columns; pitch of a token's values; state rows of a thread
  extern __shared__ __align__(16) float4 smem4[];
  float* recs = reinterpret_cast<float*>(smem4);               // two records | two value tiles [token][column] | S by columns | R, E by columns
  float* vals = recs + 2 * R::FLOATS;
  float* ss = vals + 2 * DC_T * VP;                            // pitch KP
  float* rs = ss + COLS * R::KP;                               // pitch 36
  float* es = rs + COLS * DC_TP;
  __shared__ __align__(8) unsigned long long bar_mem[2];
  const int tid = threadIdx.x, rg = dc_row(tid), cg = dc_col(tid);
  const int h = blockIdx.y, b = blockIdx.z, c0 = blockIdx.x * COLS;
  const int first = dc_first(p, b);
  const uint32_t bars = tc::smem_u32(bar_mem);
  if (tid == 0) {
    tc::mbar_init(bars, 1); tc::mbar_init(bars + 8, 1);
    tc::fence_barrier_init();
  }
  auto out_at = [&](int s, int c) { return p.o + ((size_t)(b * p.S + s) * p.H + h) * p.Dv + c; };
  for (int i = tid; i < min(first, p.S) * COLS; i += DC_THREADS)
    if (c0 + i % COLS < p.Dv) *out_at(i / COLS, c0 + i % COLS) = 0.0f;
  // state rows rg + 16 i, columns cg + 8 j
  float st[DR][TC];
  float* sbase = p.state + ((size_t)b * p.H + h) * p.D * p.Dv + c0;
#pragma unroll
  for (int i = 0; i < DR; ++i)
#pragma unroll
    for (int j = 0; j < TC; ++j) {
      const int d = rg + 16 * i, c = cg + 8 * j;
      st[i][j] = d < p.D && c0 + c < p.Dv ? sbase[(size_t)d * p.Dv + c] : 0.0f;
      ss[c * R::KP + d] = st[i][j];
    }
  const int n = (p.S - first + DC_T - 1) / DC_T;               // chunks of this row
  const float* rec0 = ws + ((size_t)b * p.H + h) * chunks * R::FLOATS;
  const float* v0 = p.u + (size_t)b * p.S * p.ldu + p.v_off + h * p.Dv + c0;
  auto fetch = [&](int c) {                                    // record and values of a chunk
    if (tid == 0) {
      const uint32_t bar = bars + 8 * (c & 1);
      tc::mbar_expect_tx(bar, R::FLOATS * 4);
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       tc::smem_u32(recs + (c & 1) * R::FLOATS)), "l"(rec0 + (size_t)c * R::FLOATS), "r"(R::FLOATS * 4), "r"(bar) : "memory");
    }
    float* dst = vals + (c & 1) * DC_T * VP;
    const int s0 = first + c * DC_T;
    if (wide) {
      for (int i = tid; i < DC_T * (COLS / 4); i += DC_THREADS) {
        const int t = i / (COLS / 4), q = i % (COLS / 4) * 4;
        const bool on = s0 + t < p.S && c0 + q < p.Dv;         // (Dv % 4 == 0)
        dc_cp16(dst + t * VP + q, on ? v0 + (size_t)(s0 + t) * p.ldu + q : p.u, on);
      }
    } else {
      for (int i = tid; i < DC_T * COLS; i += DC_THREADS) {
        const int t = i / COLS, q = i % COLS;
        dst[t * VP + q] = s0 + t < p.S && c0 + q < p.Dv ? v0[(size_t)(s0 + t) * p.ldu + q] : 0.0f;
      }
    }
  };
  __syncthreads();
  if (n > 0) fetch(0);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  for (int c = 0; c < n; ++c) {
    if (c + 1 < n) fetch(c + 1);
    const float* rec = recs + (c & 1) * R::FLOATS;
    const float* vt = vals + (c & 1) * DC_T * VP;
    tc::mbar_wait(bars + 8 * (c & 1), (c >> 1) & 1);
    // (A K) S and (A Q) S
    unsigned long long acc[4][TC] = {};
    const float* col[TC];
#pragma unroll
    for (int j = 0; j < TC; ++j) col[j] = ss + (cg + 8 * j) * R::KP;
    {
      const float* row[4] = {rec + rg * R::KP, rec + (rg + 16) * R::KP, rec + R::Q + rg * R::KP, rec + R::Q + (rg + 16) * R::KP};
      dc_dot<4, TC, D>(acc, row, col);
    }
    bool bad = false;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < TC; ++j) {
        const int t = rg + 16 * i, q = cg + 8 * j;
        const float r = vt[t * VP + q] - dc_sum2(acc[i][j]);
        bad |= !(fabsf(r) < INFINITY);
        rs[q * DC_TP + t] = r;
      }
    // A number that is not finite belongs to its token and the later ones: nothing of it may reach an earlier token through the zeros above the
    // diagonals, so such a chunk goes term by term.
    bad = __syncthreads_or(bad) != 0;
    unsigned long long eacc[2][TC] = {};
    float e[2][TC], o[2][TC];
    const float* trow[2] = {rec + R::T + rg * DC_TP, rec + R::T + (rg + 16) * DC_TP};
    const float* prow[2] = {rec + R::P + rg * DC_TP, rec + R::P + (rg + 16) * DC_TP};
    auto lower = [&](unsigned long long (&a)[2][TC], const float* const (&row)[2], const float* src) {      // row 0: its first 16 terms are all
#pragma unroll
      for (int j = 0; j < TC; ++j) col[j] = src + (cg + 8 * j) * DC_TP;
      dc_dot<2, TC, 16>(a, row, col);
      unsigned long long hi[1][TC];
      const float* hrow[1] = {row[1] + 16};
#pragma unroll
      for (int j = 0; j < TC; ++j) { hi[0][j] = a[1][j]; col[j] += 16; }
      dc_dot<1, TC, 16>(hi, hrow, col);
#pragma unroll
      for (int j = 0; j < TC; ++j) a[1][j] = hi[0][j];
    };
    if (!bad) {
      lower(eacc, trow, rs);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < TC; ++j) e[i][j] = dc_sum2(eacc[i][j]);
    } else {
      for (int i = 0; i < 2; ++i)
        for (int j = 0; j < TC; ++j) {
          float s = 0.0f;
          for (int m = 0; m <= rg + 16 * i; ++m) s = fmaf(trow[i][m], rs[(cg + 8 * j) * DC_TP + m], s);
          e[i][j] = s;
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < TC; ++j) {
        bad |= !(fabsf(e[i][j]) < INFINITY);
        es[(cg + 8 * j) * DC_TP + rg + 16 * i] = e[i][j];
      }
    bad = __syncthreads_or(bad) != 0;
    // S <- A S + (r K)^T E, then the read-outs
    {
      const float a = rec[R::A];
      unsigned long long sacc[DR][TC] = {};
      const float* krow[DR];
#pragma unroll
      for (int i = 0; i < DR; ++i) krow[i] = rec + R::KT + (rg + 16 * i) * DC_TP;
#pragma unroll
      for (int j = 0; j < TC; ++j) col[j] = es + (cg + 8 * j) * DC_TP;
      dc_dot<DR, TC, DC_T>(sacc, krow, col);
#pragma unroll
      for (int i = 0; i < DR; ++i)
#pragma unroll
        for (int j = 0; j < TC; ++j) {
          st[i][j] = fmaf(a, st[i][j], dc_sum2(sacc[i][j]));
          ss[(cg + 8 * j) * R::KP + rg + 16 * i] = st[i][j];
        }
    }
    {
      unsigned long long oacc[2][TC];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < TC; ++j) oacc[i][j] = acc[2 + i][j];
      if (!bad) lower(oacc, prow, es);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int s = first + c * DC_T + rg + 16 * i;
#pragma unroll
        for (int j = 0; j < TC; ++j) {
          const int q = c0 + cg + 8 * j;
          o[i][j] = dc_sum2(oacc[i][j]);
          if (bad)
            for (int m = 0; m <= rg + 16 * i; ++m) o[i][j] = fmaf(prow[i][m], es[(cg + 8 * j) * DC_TP + m], o[i][j]);
          if (s < p.S && q < p.Dv) *out_at(s, q) = o[i][j];
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");           // this thread's share of the next values
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < DR; ++i)
#pragma unroll
    for (int j = 0; j < TC; ++j) {
      const int d = rg + 16 * i, c = cg + 8 * j;
      if (d < p.D && c0 + c < p.Dv) sbase[(size_t)d * p.Dv + c] = st[i][j];
    }
}

bool delta_chunk_takes(int D) { return D <= 128; }
size_t delta_chunk_ws_floats(int B, int S, int H, int D) { return (size_t)B * H * ((S + DC_T - 1) / DC_T) * dc_record_floats(D); }

template <int D, int TC>
static int dc_scan(const DeltaHeadParams& p, const float* ws, int chunks, cudaStream_t st) {
  using R = DcRecord<D>;
  constexpr int COLS = 8 * TC;
  const size_t smem = (size_t)(2 * R::FLOATS + 2 * DC_T * (COLS + 8) + COLS * R::KP + 2 * COLS * DC_TP) * sizeof(float);
  const int wide = p.Dv % 4 == 0 && p.ldu % 4 == 0 && p.v_off % 4 == 0 && ((uintptr_t)p.u & 15) == 0;
  auto* kernel = delta_chunk_scan_kernel<D, TC>;
  JL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  JL_CUDA(launch_pdl(kernel, dim3((p.Dv + COLS - 1) / COLS, p.H, p.B), dim3(DC_THREADS), smem, st, p, ws, chunks, wide));
  return JL_OK;
}

template <typename T, int D>
static int dc_run(const DeltaHeadParams& p, float* ws, const void* a_bias, const void* a_log, cudaStream_t st) {
  using R = DcRecord<D>;
  const int chunks = (p.S + DC_T - 1) / DC_T;
  const size_t smem = (size_t)(2 * DC_T * R::KP + DC_T * 33 + DC_T * DC_TP + 3 * DC_T) * sizeof(float);
  auto* prep = delta_chunk_prep_kernel<T, D>;
  JL_CUDA(cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  JL_CUDA(launch_pdl(prep, dim3(chunks, p.H, p.B), dim3(DC_THREADS), smem, st, p, ws, (const T*)a_bias, (const T*)a_log));
  // Value columns of a CTA: as many as leave the SMs some three CTAs for every two of them, since a chunk is a chain of dependent steps and two CTAs hide
  // each other's.  Both launches, us, 32 | 16 | 8 columns: 2 rows x 1000 tokens x 16 heads of 64 x 128 171 | 113 | 174; 1 x 2048 of the same 307 | 205 | 174;
  // 4 x 512 x 16 heads of 128 x 128 192 | 223 | 278; 1 x 700 x 8 heads of 128 x 64 116 | 76 | 62; 8 x 2000 x 16 heads of 64 x 128 727 | 799 | 1154.
  const long rows = (long)p.B * p.H;
  if (rows * ((p.Dv + 31) / 32) >= DC_CTAS) return dc_scan<D, 4>(p, ws, chunks, st);
  if (rows * ((p.Dv + 15) / 16) >= DC_CTAS) return dc_scan<D, 2>(p, ws, chunks, st);
  return dc_scan<D, 1>(p, ws, chunks, st);
}

int delta_chunk_launch(const DeltaHeadParams& p, float* ws, const void* a_bias, const void* a_log, int dtype, cudaStream_t st) {
  if (p.D <= 32) JL_DISPATCH_DTYPE(dtype, return (dc_run<T, 32>(p, ws, a_bias, a_log, st)));
  if (p.D <= 64) JL_DISPATCH_DTYPE(dtype, return (dc_run<T, 64>(p, ws, a_bias, a_log, st)));
  JL_DISPATCH_DTYPE(dtype, return (dc_run<T, 128>(p, ws, a_bias, a_log, st)));
  return JL_OK;
}

}  // namespace jl

// Tensor-core distance + argmin in one fp16 product per (row, centroid), with an error bound and an exact pass
// over the rows the bound leaves open: float32 and float64 rows of up to 256 columns, more than 16 centroids.
//
// Replaces calculate_distances + relabel (src/gpu/kmeans/kmeans_labels.cu:115-244, kmeans_labels.h:360-392).
//
// The three-term kernels (km_assign_tc_big.cuh) spend three products to bring a score's error down to 2^-19, and
// float64 rows went to the float64 matrix unit, which is forty times slower than this one.  A label does not need
// that: the rows are rounded once to fp16 (half_rows_kernel: two bytes per element and, per row, |x|^2 and the
// length of what the rounding dropped), the scores |c|^2 - 2 x.c are formed from the rounded operands, and the
// lengths of the dropped parts bound how far the difference of two scores can be off (half_tolerance: that part is
// Cauchy-Schwarz; the tensor core's own accumulation enters with the measured constant of tol_rel_of).  A row
// whose best score is ahead of every other by more than that has its label; the others are listed with the few
// centroids that can still be nearest and settled in double precision from the unrounded rows
// (half_exact_f32_kernel, half_exact_f64_kernel).  Labels are therefore those of exact arithmetic, as before.
#pragma once

#include "km_assign_tc_big.cuh"

namespace km {
namespace tch {

using namespace km::tc;
using tcb::tc_mma_ts2;

constexpr int kNT = 128;          // centroids per accumulator
constexpr int kHalfThreads = 512; // X producer, MMA issuer, B producer, MMA issuer, 4 loader warps, 2 x 4 epilogue warps
constexpr uint32_t kPanel = 16384u;   // 128 rows or centroids x 64 columns
constexpr int kMaxK = 6144;
constexpr int kMaxD = 256;

// barriers
enum HBar { X_FULL = 0, X_EMPTY = 2, A_RDY = 4, A_EMP = 6, B_FUL = 8, B_EMP = 16, AC_FUL = 24, AC_EMP = 26, DRAIN = 28,
            NBARS = 30 };

inline int panels_of(int d) { return (d + 63) / 64; }
constexpr int x_stages(int panels) { return panels <= 2 ? 2 : 1; }
// centroid tiles (128 centroids, all columns) in flight: 128 KB of them, 96 KB for three panels
constexpr int b_stages(int panels) { return panels == 1 ? 8 : (panels == 2 ? 4 : 2); }
inline size_t half_smem_bytes(int d, int kpad) {
  const int P = panels_of(d);
  return 1024 + (size_t)(x_stages(P) + b_stages(P)) * P * kPanel + (size_t)kpad * 4 + NBARS * 8 + 64;
}

// Bound on the error of the difference between the best score of a row and any score that could belong to the
// nearest centroid, both formed as |c|^2 sx sb + xh.bh from y = x sx = xh + ey and b_j = -2 c_j sb = bh_j + eb_j:
//   (ey.b_j - ey.b_best) + (xh.eb_j - xh.eb_best) + the accumulator's own error.
// The last is what split_tolerance covers.  |xh.eb| <= |xh| max|eb| for each of the two.  And for the true
// nearest centroid j, |c_j - c_best| <= 2 |x - c_best|, so the first is at most |ey| 2 sb 2 |x - c_best|, with
// |x - c_best|^2 = |x|^2 + score taken from the computed score plus its own error.  All lengths are known: |ey| per
// row, max|eb| per table, both of the rounding as it happened (no assumption on subnormals).
__device__ __forceinline__ float half_tolerance(float tol_rel, float tol_floor, float xn, float ey, float best,
                                                float cn_max, float eb_max, float sx, float sxsb) {
  const float t3 = split_tolerance(tol_rel, tol_floor, xn, cn_max, sx, sxsb);
  const float sb2 = 2.0f * sxsb / sx;
  const float errb = (sx * sqrtf(xn) + ey) * eb_max;
  const float single = t3 + errb + ey * sb2 * sqrtf(cn_max);
  const float dist_sq = xn + (best + single) / sxsb;
  return t3 + 1.001f * (2.0f * errb + 2.0f * ey * sb2 * sqrtf(fmaxf(dist_sq, 0.f)));
}

// Rows rounded to fp16: xh [rows][ldh] (columns d .. ldh zero; ldh = d rounded up to eight, what TMA can address),
// rowq[row] = (|x|^2, |x sx - xh|).  `lpr` lanes (a power of two) share a row, four consecutive columns per lane and
// step.  Bound by HBM: reads sizeof(T) and writes two bytes per element.
template <typename T> struct Quad;
template <> struct Quad<float> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[4]) {
    const float4 q = __ldcs(reinterpret_cast<const float4*>(p));
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  }
};
template <> struct Quad<double> {
  static __device__ __forceinline__ void load(const double* p, double (&v)[4]) {
    const double2 a = __ldcs(reinterpret_cast<const double2*>(p));
    const double2 b = __ldcs(reinterpret_cast<const double2*>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
};

template <typename T, bool VEC>
__global__ void __launch_bounds__(256)
half_rows_kernel(const T* __restrict__ X, size_t n, int d, int ldh, int lpr, float sx, __half* __restrict__ xh,
                 float2* __restrict__ rowq) {
  constexpr int U = sizeof(T) == 8 ? 4 : 8;
  const int lane = threadIdx.x & 31;
  const int rpw = 32 / lpr, g = lane / lpr, l = lane % lpr;
  const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const size_t nwarp = ((size_t)gridDim.x * blockDim.x) >> 5;
  const T s = (T)sx;
  for (size_t base = warp * rpw * U; base < n; base += nwarp * rpw * U) {
    T q[U], e[U];
#pragma unroll
    for (int u = 0; u < U; ++u) { q[u] = (T)0; e[u] = (T)0; }
    for (int t0 = l * 4; t0 - l * 4 < ldh; t0 += lpr * 4) {
      T v[U][4];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const size_t row = base + (size_t)u * rpw + g;
#pragma unroll
        for (int c = 0; c < 4; ++c) v[u][c] = (T)0;
        if (row < n && t0 < d) {
          const T* p = X + row * (size_t)d + t0;
          if (VEC) {                     // d is a multiple of four, rows are 16-byte aligned
            Quad<T>::load(p, v[u]);
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
              if (t0 + c < d) v[u][c] = p[c];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const size_t row = base + (size_t)u * rpw + g;
        __half h[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const T y = v[u][c] * s;
          h[c] = to_half(y);
          const T r = y - (T)__half2float(h[c]);   // exact
          q[u] = fma(v[u][c], v[u][c], q[u]);
          e[u] = fma(r, r, e[u]);
        }
        if (row < n && t0 < ldh) {
          const __half2 a = __halves2half2(h[0], h[1]), b = __halves2half2(h[2], h[3]);
          *reinterpret_cast<uint2*>(xh + row * (size_t)ldh + t0) =
              make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      for (int o = lpr >> 1; o > 0; o >>= 1) {
        q[u] += __shfl_xor_sync(0xffffffffu, q[u], o);
        e[u] += __shfl_xor_sync(0xffffffffu, e[u], o);
      }
      const size_t row = base + (size_t)u * rpw + g;
      // the sums' own rounding is far below the margin: 1e-4 on |ey|, the relative term of split_tolerance for |x|^2
      if (row < n && l == 0) rowq[row] = make_float2((float)q[u], 1.0001f * sqrtf((float)e[u]) + 1e-30f);
    }
  }
}

// Bound by the tensor pipe at 256 columns (92 % of its cycles; 1.54 PFLOP/s, a library GEMM 1.69), below that by the
// hand-over of the accumulator between the MMAs and the epilogue (128 columns: 1.0, 64: 0.56 PFLOP/s).  2e6 x 128 rows
// with 1000 centroids: 0.48 ms per pass (three-term kernel 1.20), 5e5 x 256 with 4096: 0.68 (2.12), 60,000 x 256
// float64 rows with 4096: 0.10 (float64 matrix unit 5.7).  What made the three-term kernel's layout unfit:
//   * with a third of the MMAs per centroid the centroid panels would have to come from L2 three times as fast (64
//     bytes per clock and SM), so a CTA works on two row tiles at a time: every panel that arrives is used twice;
//   * its fold of a score takes longer than the product.  Here no index is carried: a score's column is (chunk of 32,
//     position in the chunk).  Per position the minimum over all chunks, per chunk the minimum over its positions, the
//     three smallest of those with their chunks and the value of the fourth.  Another score within the bound lies in
//     another chunk, or in the same chunk at another position, so either shows.  At the end of a row the positions
//     (a 32-bit mask) and the chunks within the bound are the candidates for the exact pass;
//   * an MMA took longer to issue (115 clocks: see elect_one) than to run (64), and each satisfied wait takes about
//     200 clocks: the issuing warps stay converged, poll their barriers side by side, and each row tile has its own.
// A operand in TMEM (2 tiles x up to 128 columns), one accumulator of 128 columns per row tile.  Tried instead: three
// accumulators shared by both tiles with one issuer (1.23 PFLOP/s at 256 columns, 0.85 at 128), both operands from
// shared memory and two accumulators per tile (1.10 and 1.0: shared memory delivers 128 bytes per clock, all that
// such MMAs take), 16 epilogue warps with a row's columns cut in two (no difference, and spills).
// Every barrier has one waiter that takes its phases in order, except the centroid tiles' "full" barrier: a phase of
// it can only end after both issuers have handed the tile back, so neither can miss one.
template <int P>   // 64-column panels of a row
__global__ void __launch_bounds__(kHalfThreads, 1)
assign_tc_half_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmB,
                      const float* __restrict__ cn_pad, const float2* __restrict__ rowq, int* __restrict__ labels,
                      size_t n, int n_sub, int kpad, int ksteps, IterState* st, int count_changes,
                      uint4* __restrict__ cand_near, unsigned int cand_cap,
                      unsigned int all_limit, float tol_rel, float tol_floor, float sx, float sxsb,
                      unsigned int wait_iters, unsigned int* host_whole) {
  if (st->full_rows) {   // this matrix left too many rows open before: the kernel behind this one has the pass
    if (host_whole && blockIdx.x == 0 && threadIdx.x == 0) *host_whole = 1;
    return;
  }
  constexpr int NX = x_stages(P), NB = b_stages(P);
  constexpr uint32_t kXBytes = P * kPanel;
  constexpr uint32_t kAccCol = 2u * P * 32u;     // accumulators behind the two A buffers
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_u32 = smem_u32(smem_raw);
  const uint32_t base = (raw_u32 + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw_u32);

  constexpr uint32_t off_b = NX * kXBytes;
  constexpr uint32_t off_cn = off_b + NB * kXBytes;
  const uint32_t off_bar = off_cn + (uint32_t)kpad * 4u;
  const uint32_t off_misc = off_bar + NBARS * 8;
  float* cn_s = reinterpret_cast<float*>(sm + off_cn);
  volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(sm + off_misc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + off_misc + 4);
  auto bar = [&](int i) { return base + off_bar + (uint32_t)i * 8u; };

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int n_ct = kpad / kNT;
  // this CTA's 128-row tiles
  const int s_begin = (int)((long long)blockIdx.x * n_sub / gridDim.x);
  const int s_end = (int)((long long)(blockIdx.x + 1) * n_sub / gridDim.x);

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(X_FULL + i), 1);
      mbar_init(bar(X_EMPTY + i), 128);
      mbar_init(bar(A_RDY + i), 128);
      mbar_init(bar(A_EMP + i), 1);
    }
    for (int s = 0; s < NB; ++s) { mbar_init(bar(B_FUL + s), 1); mbar_init(bar(B_EMP + s), 2); }
    for (int a = 0; a < 2; ++a) { mbar_init(bar(AC_FUL + a), 1); mbar_init(bar(AC_EMP + a), 128); }
    for (int a = 0; a < 2; ++a) mbar_init(bar(DRAIN + a), 1);
    *abort_flag = 0;
    abort_flag[3] = (int)wait_iters;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < kpad; i += kHalfThreads) cn_s[i] = cn_pad[i];
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(base + off_misc),
                 "r"((uint32_t)kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_holder, 0);   // known to be uniform
  const float cn_max = cn_pad[kpad], eb_max = cn_pad[kpad + 1];
  const uint32_t idesc = (1u << 4) | ((uint32_t)(kNT >> 3) << 17) | ((128u >> 4) << 24);

  if (warp == 0) {
    // ------------------------------ X producer: one 128-row tile per step ------------------------------
    if (lane == 0) {
      int xi = 0;
      bool ok = true;
      for (int s = s_begin; s < s_end; ++s, ++xi) {
        const int b = xi % NX;
        if (xi >= NX) ok = mbar_wait(bar(X_EMPTY + b), (uint32_t)(xi / NX - 1) & 1u, abort_flag, 1);
        if (!ok) break;
        mbar_expect_tx(bar(X_FULL + b), kXBytes);
#pragma unroll
        for (int p = 0; p < P; ++p)
          tma_load_2d(base + (uint32_t)b * kXBytes + p * kPanel, &tmX, p * 64, s * kBM, bar(X_FULL + b));
      }
      if (!ok)
        for (int j = (xi > NX ? xi - NX : 0); j < xi; ++j) mbar_drain(bar(X_FULL + j % NX), (uint32_t)(j / NX) & 1u);
    }
  } else if (warp == 2) {
    // ------------------------------ centroid tiles ------------------------------
    if (lane == 0) {
      int bs = 0;
      bool ok = true;
      for (int s = s_begin; s < s_end && ok; s += 2) {
        for (int ct = 0; ct < n_ct; ++ct, ++bs) {
          const int b = bs % NB;
          if (bs >= NB) ok = mbar_wait(bar(B_EMP + b), (uint32_t)(bs / NB - 1) & 1u, abort_flag, 2);
          if (!ok) break;
          mbar_expect_tx(bar(B_FUL + b), kXBytes);
#pragma unroll
          for (int p = 0; p < P; ++p)
            tma_load_2d(base + off_b + (uint32_t)b * kXBytes + p * kPanel, &tmB, p * 64, ct * kNT, bar(B_FUL + b));
        }
      }
      if (!ok)
        for (int j = (bs > NB ? bs - NB : 0); j < bs; ++j) mbar_drain(bar(B_FUL + j % NB), (uint32_t)(j / NB) & 1u);
    }
  } else if (warp == 1 || warp == 3) {
    // ------------------------------ MMA issuers, one per row tile of the pair ------------------------------
    // the warp stays converged and one elected lane issues
    const int sub = warp >> 1;
    bool ok = true;
    int it = 0, bs = 0, u = 0;
    const uint32_t desc_hi = (uint32_t)(smem_desc_sw128(0) >> 32);
    const int k_last = ksteps - 4 * (P - 1);
    auto wait = [&](int b, uint32_t parity, int code) {
      return __all_sync(0xffffffffu, mbar_wait(bar(b), parity, abort_flag, code)) != 0;
    };
    const uint32_t a_base = tmem_base + (uint32_t)sub * (P * 32u);
    for (int s = s_begin; s < s_end && ok; s += 2, ++it) {
      const bool have = s + sub < s_end;
      for (int ct = 0; ct < n_ct && ok; ++ct, ++bs) {
        const int b = bs % NB;
        if (!have) {   // no second tile: only hand the centroid tile back
          ok = wait(B_FUL + b, (uint32_t)(bs / NB) & 1u, 5);
          if (ok && lane == 0) mbar_arrive(bar(B_EMP + b));
          continue;
        }
        if (ct == 0) ok = wait(A_RDY + sub, (uint32_t)it & 1u, 3);
        {
          // both barriers polled side by side: a satisfied wait still takes about 200 clocks
          const bool t1 = u == 0 || mbar_try(bar(AC_EMP + sub), (uint32_t)(u - 1) & 1u);
          const bool t2 = mbar_try(bar(B_FUL + b), (uint32_t)(bs / NB) & 1u);
          if (ok && !__all_sync(0xffffffffu, t1 && t2)) {
            if (u > 0) ok = wait(AC_EMP + sub, (uint32_t)(u - 1) & 1u, 4);
            if (ok) ok = wait(B_FUL + b, (uint32_t)(bs / NB) & 1u, 5);
          }
        }
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          const uint32_t acc = tmem_base + kAccCol + (uint32_t)sub * kNT;
          const uint32_t lo = (uint32_t)smem_desc_sw128(base + off_b + (uint32_t)b * kXBytes);
#pragma unroll
          for (int p = 0; p < P; ++p) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              if (p < P - 1 || kk < k_last)
                tc_mma_ts2(acc, a_base + (uint32_t)(p * 4 + kk) * 8u, lo + (uint32_t)(p * (kPanel >> 4) + kk * 2),
                           desc_hi, idesc, (p | kk) ? 1u : 0u);
          }
          tc_commit(bar(AC_FUL + sub));
          tc_commit(bar(B_EMP + b));
          if (ct == n_ct - 1) tc_commit(bar(A_EMP + sub));
        }
        __syncwarp();
        ++u;
      }
    }
    if (!ok) {
      // every MMA issued so far must retire before TMEM is freed
      if (elect_one()) tc_commit(bar(DRAIN + sub));
      __syncwarp();
      mbar_drain(bar(DRAIN + sub), 0);
    }
  } else if (warp < 8) {
    // ------------------------------ loader: row tile from shared memory into the A buffer ------------------------------
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    bool ok = true;
    int xi = 0, it = 0;
    for (int s = s_begin; s < s_end && ok; s += 2, ++it) {
      const int nsub = (s + 1 < s_end) ? 2 : 1;
      for (int sub = 0; sub < nsub && ok; ++sub, ++xi) {
        const int b = xi % NX;
        ok = mbar_wait(bar(X_FULL + b), (uint32_t)(xi / NX) & 1u, abort_flag, 6);
        if (ok && it >= 1) ok = mbar_wait(bar(A_EMP + sub), (uint32_t)(it - 1) & 1u, abort_flag, 7);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t dst = tmem_base + lane_addr + (uint32_t)sub * (P * 32u);
#pragma unroll
        for (int p = 0; p < P; ++p) {
          const uint8_t* rowp = sm + (uint32_t)b * kXBytes + p * kPanel + row * 128;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t v[16];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const uint4 w = *reinterpret_cast<const uint4*>(rowp + (((half * 4 + c) ^ (row & 7)) << 4));
              v[c * 4 + 0] = w.x; v[c * 4 + 1] = w.y; v[c * 4 + 2] = w.z; v[c * 4 + 3] = w.w;
            }
            tmem_st16(dst + (uint32_t)(p * 32 + half * 16), v);
          }
        }
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(bar(X_EMPTY + b));
        mbar_arrive(bar(A_RDY + sub));
      }
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    const int grp = (warp - 8) >> 2;        // row tile of the pair
    const int q = warp & 3;
    const int row_in_tile = q * 32 + lane;
    const uint32_t acc0 = tmem_base + ((uint32_t)(q * 32) << 16) + kAccCol +
                         (uint32_t)grp * kNT;
    const float kInf = __int_as_float(0x7f800000);
    unsigned int changed = 0;
    bool ok = true;
    int u = 0;              // units (accumulator fills) of this group
    for (int s = s_begin; s < s_end && ok; s += 2) {
      const int nsub = (s + 1 < s_end) ? 2 : 1;
      if (grp >= nsub) break;
      const size_t row = (size_t)(s + grp) * kBM + row_in_tile;
      float2 xq = make_float2(0.f, 0.f);
      int old_label = -1;
      if (row < n) {
        xq = __ldcs(rowq + row);
        if (count_changes) old_label = labels[row];
      }
      float b1 = kInf, b2 = kInf, b3 = kInf, b4 = kInf;
      uint32_t i1 = 0xffffu, i2 = 0xffffu, i3 = 0xffffu;
      float colmin[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) colmin[i] = kInf;
      for (int ct = 0; ct < n_ct; ++ct) {
        ok = mbar_wait(bar(AC_FUL + grp), (uint32_t)u & 1u, abort_flag, 8);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const float* cnp = cn_s + ct * kNT;
        // a chunk's 32 scores; the next chunk is on its way from TMEM meanwhile
        auto fold = [&](const uint32_t (&v)[32], int ch) {
          float sc[32];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float4 c4 = *reinterpret_cast<const float4*>(cnp + ch * 32 + i * 4);
            sc[i * 4 + 0] = __uint_as_float(v[i * 4 + 0]) + c4.x;
            sc[i * 4 + 1] = __uint_as_float(v[i * 4 + 1]) + c4.y;
            sc[i * 4 + 2] = __uint_as_float(v[i * 4 + 2]) + c4.z;
            sc[i * 4 + 3] = __uint_as_float(v[i * 4 + 3]) + c4.w;
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) colmin[i] = fminf(colmin[i], sc[i]);
          float t[11];
#pragma unroll
          for (int i = 0; i < 10; ++i) t[i] = fmin3(sc[3 * i], sc[3 * i + 1], sc[3 * i + 2]);
          t[10] = fminf(sc[30], sc[31]);
          const float m = fminf(fmin3(fmin3(t[0], t[1], t[2]), fmin3(t[3], t[4], t[5]), fmin3(t[6], t[7], t[8])),
                                fminf(t[9], t[10]));
          const uint32_t id = (uint32_t)(ct * 4 + ch);
          const bool l1 = m < b1, l2 = m < b2, l3 = m < b3;
          b4 = fminf(b4, fmaxf(m, b3));
          b3 = fminf(b3, fmaxf(m, b2));
          b2 = fminf(b2, fmaxf(m, b1));
          b1 = fminf(b1, m);
          i3 = l2 ? i2 : (l3 ? id : i3);
          i2 = l1 ? i1 : (l2 ? id : i2);
          i1 = l1 ? id : i1;
        };
        uint32_t va[32], vb[32];
        tmem_ld16(acc0, va, 0);
        tmem_ld16(acc0 + 16, va, 16);
        tmem_wait_ld(va);
        tmem_ld16(acc0 + 32, vb, 0);
        tmem_ld16(acc0 + 48, vb, 16);
        fold(va, 0);
        tmem_wait_ld(vb);
        tmem_ld16(acc0 + 64, va, 0);
        tmem_ld16(acc0 + 80, va, 16);
        fold(vb, 1);
        tmem_wait_ld(va);
        tmem_ld16(acc0 + 96, vb, 0);
        tmem_ld16(acc0 + 112, vb, 16);
        fold(va, 2);
        tmem_wait_ld(vb);
        // the accumulator is in registers: the MMAs may have it back
        tc_fence_before();
        mbar_arrive(bar(AC_EMP + grp));
        fold(vb, 3);
        ++u;
      }
      if (!ok) break;
      const float lim = b1 + half_tolerance(tol_rel, tol_floor, xq.x, xq.y, b1, cn_max, eb_max, sx, sxsb);
      uint32_t mask = 0;
#pragma unroll
      for (int i = 0; i < 32; ++i) mask |= (colmin[i] <= lim) ? (1u << i) : 0u;
      bool open = false;
      if (row < n) {
        // no other chunk and no other position within the bound: the label is certain (a bound that is no number
        // leaves the mask empty)
        if (__popc(mask) == 1 && b2 > lim) {
          const int label = (int)(i1 * 32u) + __ffs((int)mask) - 1;
          changed += (old_label != label);
          labels[row] = label;
        } else {
          open = true;
        }
      }
      const unsigned int vote = __ballot_sync(0xffffffffu, open);
      if (vote) {
        // .x: positions within the bound; .y/.z: chunks, 0xffff = none; high half of .z: 1 = any chunk may hold the
        // nearest centroid
        const bool all = b4 <= lim || !(b1 <= lim);
        const unsigned int vall = __ballot_sync(0xffffffffu, open && all);
        unsigned int pos = 0;
        if (lane == 0) {
          pos = atomicAdd(&st->cand_count, (unsigned int)__popc(vote));
          if (vall) atomicAdd(&st->cand_all, (unsigned int)__popc(vall));
        }
        pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(vote & ((1u << lane) - 1u));
        // rows beyond the list's end are not lost: the count then sends the whole pass to the kernel behind
        if (open && pos < cand_cap)
          cand_near[pos] = make_uint4(mask ? mask : 0xffffffffu, i1 | ((b2 <= lim ? i2 : 0xffffu) << 16),
                                      (b3 <= lim ? i3 : 0xffffu) | (all ? 0x10000u : 0u), (uint32_t)row);
      }
    }
    if (count_changes) {
      changed = __reduce_add_sync(0xffffffffu, changed);
      if (lane == 0 && changed) atomicAdd(&st->changed, (unsigned long long)changed);
    }
  }

  __syncthreads();
  if (tid == 0) {
    if (*abort_flag) atomicMax(&st->error, *abort_flag);
    // the CTA that finishes last decides whether the exact pass settles the open rows or the pass is repeated by
    // the kernel behind this one, which needs no list (labels written here stay right: it only repeats them)
    __threadfence();
    if (atomicAdd(&st->half_done, 1u) == gridDim.x - 1) {
      __threadfence();
      st->half_done = 0;
      const unsigned int cand = atomicAdd(&st->cand_count, 0u), all = atomicAdd(&st->cand_all, 0u);
      st->cand_all = 0;
      const bool whole = cand > cand_cap || all > all_limit;
      if (whole) {
        st->full_rows = 1;
        st->cand_count = 0;
      }
      if (host_whole) *host_whole = whole ? 1 : 0;
    }
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kTmemCols)
                 : "memory");
  }
}

// Rows of which every chunk may hold the nearest centroid (k / 32 times the work of the others) are put by and
// settled by all warps of the CTA together, in double precision, once the others are done: left to one warp each, a
// handful of them took longer than everything else (4096 centroids: 100 us for 500 rows).
constexpr int kExactWarps = 8;
constexpr int kPutBy = 64;       // per CTA; further ones are settled by their warp
struct PutBy {
  uint4 rec[kPutBy];
  unsigned int n;
  double best[kExactWarps];
  int idx[kExactWarps];
};
// true: the row has been put by
__device__ __forceinline__ bool put_by(PutBy& pb, const uint4& rec, int lane) {
  unsigned int at = 0;
  if (lane == 0) at = atomicAdd(&pb.n, 1u);
  at = __shfl_sync(0xffffffffu, at, 0);
  if (at >= kPutBy) return false;
  if (lane == 0) pb.rec[at] = rec;
  return true;
}
template <typename T>
__device__ __forceinline__ unsigned int settle_put_by(PutBy& pb, unsigned char* pos, const T* __restrict__ X, int d,
                                                      const double* __restrict__ Cd, int k, int kpad,
                                                      int* __restrict__ labels) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 3, l = lane & 7;
  unsigned int changed = 0;
  __syncthreads();
  const unsigned int n = min(pb.n, (unsigned int)kPutBy);
  for (unsigned int e = 0; e < n; ++e) {
    const uint4 rec = pb.rec[e];
    const T* xr = X + (size_t)rec.w * d;
    if ((rec.x >> lane) & 1u) pos[__popc(rec.x & ((1u << lane) - 1u))] = (unsigned char)lane;
    __syncwarp();
    const int n_pos = __popc(rec.x), total = kpad / 32 * n_pos;
    double best = __longlong_as_double(0x7ff0000000000000LL);
    int bi = 0x7fffffff;
    for (int m0 = warp * 4; m0 < total; m0 += kExactWarps * 4) {
      const int m = m0 + g, ch = m / n_pos;
      const int c = m < total ? ch * 32 + pos[m - ch * n_pos] : k;
      double s = 0.0;
      if (c < k) {
        const double* cr = Cd + (size_t)c * d;
#pragma unroll 8
        for (int t = l; t < d; t += 8) { const double q = widen_exact(xr[t]) - cr[t]; s = fma(q, q, s); }
      }
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      if (c < k && (s < best || (s == best && c < bi))) { best = s; bi = c; }
    }
#pragma unroll
    for (int o = 16; o >= 8; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob < best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if (lane == 0) { pb.best[warp] = best; pb.idx[warp] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < kExactWarps; ++w)
        if (pb.best[w] < best || (pb.best[w] == best && pb.idx[w] < bi)) { best = pb.best[w]; bi = pb.idx[w]; }
      if (bi != 0x7fffffff) {
        changed += (labels[rec.w] != bi);
        labels[rec.w] = bi;
      }
    }
    __syncthreads();
  }
  return changed;
}

// Settles the listed float64 rows: squared distances to the recorded candidates as direct differences in double precision
// from the unrounded rows and centroids, smallest wins, lowest index on a tie.  A warp takes a row, eight lanes a
// candidate (chunk x position), so four are looked at side by side: the pass is bound by the latency of the
// candidates' rows from L2 (d * 8 bytes each) and of the double-precision reductions, not by their throughput.
__global__ void __launch_bounds__(kExactWarps * 32)
half_exact_f64_kernel(const double* __restrict__ X, int d, const double* __restrict__ Cd, int k, int kpad,
                  const uint4* __restrict__ cand_near, IterState* st, int* __restrict__ labels, int count_changes) {
  __shared__ __align__(16) double xs_all[kExactWarps][kMaxD];
  __shared__ unsigned char pos_all[kExactWarps][32];
  __shared__ PutBy pb;
  if (threadIdx.x == 0) pb.n = 0;
  __syncthreads();
  const unsigned int cnt = st->cand_count;
  const int lane = threadIdx.x & 31;
  double* xs = xs_all[threadIdx.x >> 5];
  unsigned char* pos = pos_all[threadIdx.x >> 5];
  const unsigned int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned int nwarp = (gridDim.x * blockDim.x) >> 5;
  const int g = lane >> 3, l = lane & 7;
  unsigned int changed = 0;
  uint4 r = make_uint4(0, 0, 0, 0);
  if (warp < cnt) r = cand_near[warp];
  for (unsigned int e = warp; e < cnt; e += nwarp) {
    const uint4 rec = r;
    if (e + nwarp < cnt) r = cand_near[e + nwarp];   // the next row's record is on its way
    const bool all = (rec.z >> 16) != 0;
    if (all && put_by(pb, rec, lane)) continue;
    const size_t row = rec.w;
    for (int t = lane; t < d; t += 32) xs[t] = X[row * (size_t)d + t];
    if ((rec.x >> lane) & 1u) pos[__popc(rec.x & ((1u << lane) - 1u))] = (unsigned char)lane;
    __syncwarp();
    const int n_pos = __popc(rec.x);
    const unsigned int id0 = rec.y & 0xffffu, id1 = rec.y >> 16, id2 = rec.z & 0xffffu;
    const int n_chunk = all ? kpad / 32 : (id2 != 0xffffu ? 3 : (id1 != 0xffffu ? 2 : 1));
    double best = __longlong_as_double(0x7ff0000000000000LL);
    int bi = 0x7fffffff;
    for (int m0 = 0; m0 < n_chunk * n_pos; m0 += 4) {
      const int m = m0 + g;
      const int ch = m / n_pos;
      int c = k;
      if (ch < n_chunk) c = (int)(all ? (unsigned int)ch : (ch == 0 ? id0 : (ch == 1 ? id1 : id2))) * 32 + pos[m - ch * n_pos];
      double s = 0.0;
      if (c < k) {
        const double* cr = Cd + (size_t)c * d;
#pragma unroll 8
        for (int t = l; t < d; t += 8) { const double q = xs[t] - cr[t]; s = fma(q, q, s); }
      }
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      if (c < k && (s < best || (s == best && c < bi))) { best = s; bi = c; }
    }
#pragma unroll
    for (int o = 16; o >= 8; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob < best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if (lane == 0 && bi != 0x7fffffff) {
      changed += (labels[row] != bi);
      labels[row] = bi;
    }
    __syncwarp();
  }
  changed += settle_put_by<double>(pb, pos, X, d, Cd, k, kpad, labels);
  if (count_changes && lane == 0 && changed) atomicAdd(&st->changed, (unsigned long long)changed);
}

// The same for float32 rows, where single precision settles nearly all of them: a sum of d squared direct differences
// formed in single precision is within (d + 2) 2^-24 of its value (all terms are positive, every operation rounds
// once), so a candidate that is ahead by more than twice that is the nearest one.  The others - and rows whose
// squares leave the range of normal numbers - are formed again in double precision.  Eight lanes share a candidate,
// four consecutive columns per lane and step (VEC: d a multiple of four, 16-byte aligned rows), NI steps.
template <int NI, bool VEC>
__global__ void __launch_bounds__(kExactWarps * 32)
half_exact_f32_kernel(const float* __restrict__ X, int d, const float* __restrict__ C, const double* __restrict__ Cd,
                      int k, int kpad, const uint4* __restrict__ cand_near, IterState* st, int* __restrict__ labels,
                      int count_changes) {
  __shared__ unsigned char pos_all[kExactWarps][32];
  __shared__ PutBy pb;
  if (threadIdx.x == 0) pb.n = 0;
  __syncthreads();
  const unsigned int cnt = st->cand_count;
  const int lane = threadIdx.x & 31;
  unsigned char* pos = pos_all[threadIdx.x >> 5];
  const unsigned int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned int nwarp = (gridDim.x * blockDim.x) >> 5;
  const int g = lane >> 3, l = lane & 7;
  const float kInf = __int_as_float(0x7f800000);
  const float ahead = 1.0f + 2.1f * (float)(d + 2) * 5.9604645e-8f;
  auto col = [&](int i, int c) { return VEC ? l * 4 + 32 * i + c : l + 8 * (4 * i + c); };
  auto fetch = [&](const float* p, float (&v)[NI][4]) {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      if (VEC) {
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (col(i, 0) < d) q = *reinterpret_cast<const float4*>(p + col(i, 0));
        v[i][0] = q.x; v[i][1] = q.y; v[i][2] = q.z; v[i][3] = q.w;
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) v[i][c] = col(i, c) < d ? p[col(i, c)] : 0.f;
      }
    }
  };
  unsigned int changed = 0;
  uint4 r = make_uint4(0, 0, 0, 0);
  if (warp < cnt) r = cand_near[warp];
  for (unsigned int e = warp; e < cnt; e += nwarp) {
    const uint4 rec = r;
    if (e + nwarp < cnt) r = cand_near[e + nwarp];   // the next row's record is on its way
    const bool all = (rec.z >> 16) != 0;
    if (all && put_by(pb, rec, lane)) continue;
    const size_t row = rec.w;
    float x[NI][4];
    fetch(X + row * (size_t)d, x);
    int old_label = -1;
    if (lane == 0) old_label = labels[row];
    if ((rec.x >> lane) & 1u) pos[__popc(rec.x & ((1u << lane) - 1u))] = (unsigned char)lane;
    __syncwarp();
    const int n_pos = __popc(rec.x);
    const unsigned int id0 = rec.y & 0xffffu, id1 = rec.y >> 16, id2 = rec.z & 0xffffu;
    const int n_chunk = all ? kpad / 32 : (id2 != 0xffffu ? 3 : (id1 != 0xffffu ? 2 : 1));
    auto candidate = [&](int m) {
      const int ch = m / n_pos;
      if (ch >= n_chunk) return k;
      return (int)(all ? (unsigned int)ch : (ch == 0 ? id0 : (ch == 1 ? id1 : id2))) * 32 + pos[m - ch * n_pos];
    };
    float best = kInf, second = kInf;
    int bi = 0x7fffffff;
    for (int m0 = 0; m0 < n_chunk * n_pos; m0 += 4) {
      const int c = candidate(m0 + g);
      float s = 0.f;
      if (c < k) {
        float v[NI][4];
        fetch(C + (size_t)c * d, v);
        float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < NI; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) { const float q = x[i][j] - v[i][j]; a[j] = fmaf(q, q, a[j]); }
        s = (a[0] + a[1]) + (a[2] + a[3]);
      }
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      if (c < k) {
        second = fminf(second, fmaxf(s, best));
        if (s < best) { best = s; bi = c; }
      }
    }
#pragma unroll
    for (int o = 16; o >= 8; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o), os = __shfl_xor_sync(0xffffffffu, second, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      second = fminf(fminf(second, os), fmaxf(best, ob));
      if (ob < best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if (!(second > best * ahead + 1e-34f)) {   // the same in every lane
      double bestd = __longlong_as_double(0x7ff0000000000000LL);
      bi = 0x7fffffff;
      for (int m0 = 0; m0 < n_chunk * n_pos; m0 += 4) {
        const int c = candidate(m0 + g);
        double s = 0.0;
        if (c < k) {
          const float* xr = X + row * (size_t)d;
          const double* cr = Cd + (size_t)c * d;
#pragma unroll 4
          for (int t = l; t < d; t += 8) { const double q = widen_exact(xr[t]) - cr[t]; s = fma(q, q, s); }
        }
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if (c < k && (s < bestd || (s == bestd && c < bi))) { bestd = s; bi = c; }
      }
#pragma unroll
      for (int o = 16; o >= 8; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, bestd, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob < bestd || (ob == bestd && oi < bi)) { bestd = ob; bi = oi; }
      }
    }
    if (lane == 0 && bi != 0x7fffffff) {
      changed += (old_label != bi);
      labels[row] = bi;
    }
    __syncwarp();
  }
  changed += settle_put_by<float>(pb, pos, X, d, Cd, k, kpad, labels);
  if (count_changes && lane == 0 && changed) atomicAdd(&st->changed, (unsigned long long)changed);
}

}  // namespace tch
}  // namespace km

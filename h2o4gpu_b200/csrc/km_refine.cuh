// Exact re-evaluation of ambiguous rows (tensor-core path for small centroid tables).
//
// The fast kernel hands over every row that has more than one score within the error bound of its best
// score, together with the bit mask of those columns (128 bits, one per centroid).  The true nearest
// centroid is one of them - every other score is farther than the bound - so only those few squared
// distances are formed again, as direct differences in double precision, and the smallest is taken, lowest
// index first on a tie.  Labels then agree with exact arithmetic on the float inputs.
//
// D / 4 lanes share a row (a float4 of it each), so a warp works on 2 (D = 64) or 4 rows at a time; x is
// widened once with integer operations and the centroids are read from the table in double, because
// float -> double conversions run at a small fraction of the FMA rate.  The list has one segment per CTA of
// the fast kernel; kRefineSplit CTAs share a segment.  Bound by the scattered reads of the listed rows
// (D * 4 bytes each): 316,000 of 1e7 x 64 rows in 53 us.
#pragma once

#include "km_common.cuh"

namespace km {

constexpr int kRefineThreads = 256;
constexpr int kRefineSplit = 6;

template <int D>
__global__ void __launch_bounds__(kRefineThreads)
refine_near_kernel(const float* __restrict__ X, const double* __restrict__ Cd, int k,
                   const unsigned int* __restrict__ amb_rows, const uint4* __restrict__ amb_near,
                   const unsigned int* __restrict__ amb_seg, unsigned int seg_cap, int n_seg, IterState* st,
                   int* __restrict__ labels, int count_changes, unsigned int* __restrict__ moved_bits) {
  constexpr int L = D / 4;                          // lanes per row
  constexpr int R = kRefineThreads / L;             // rows per CTA and step
  const int seg = blockIdx.x % n_seg;
  const unsigned int cnt = amb_seg[seg];
  const unsigned int* rows = amb_rows + (size_t)seg * seg_cap;
  const uint4* nears = amb_near + (size_t)seg * seg_cap;
  const int l = threadIdx.x % L;
  const unsigned int g = threadIdx.x / L;
  unsigned int changed = 0;
  for (unsigned int e0 = (blockIdx.x / n_seg) * R; e0 < cnt; e0 += R * kRefineSplit) {
    const bool have = e0 + g < cnt;
    size_t row = 0;
    int old_label = -1;
    unsigned long long m0 = 0, m1 = 0;
    double x[4] = {0.0, 0.0, 0.0, 0.0};
    if (have) {
      row = rows[e0 + g];
      const uint4 nm = nears[e0 + g];
      m0 = nm.x | ((unsigned long long)nm.y << 32);
      m1 = nm.z | ((unsigned long long)nm.w << 32);
      const float4 v = reinterpret_cast<const float4*>(X + row * D)[l];
      if (l == 0) old_label = labels[row];
      x[0] = widen_exact(v.x); x[1] = widen_exact(v.y); x[2] = widen_exact(v.z); x[3] = widen_exact(v.w);
    }
    double best = __longlong_as_double(0x7ff0000000000000LL);
    int bi = 0x7fffffff;
    // the rows of a warp step through their candidates together (ascending, so a strict comparison keeps the
    // lowest index on a tie)
    while (__any_sync(0xffffffffu, (m0 | m1) != 0)) {
      int c = -1;
      if (m0) { c = __ffsll((long long)m0) - 1; m0 &= m0 - 1; }
      else if (m1) { c = 64 + __ffsll((long long)m1) - 1; m1 &= m1 - 1; }
      double s = 0.0;
      if (c >= 0 && c < k) {
        const double2* cr = reinterpret_cast<const double2*>(Cd + (size_t)c * D) + 2 * l;
        const double2 a = cr[0], b = cr[1];
        const double q0 = x[0] - a.x, q1 = x[1] - a.y, q2 = x[2] - b.x, q3 = x[3] - b.y;
        s = fma(q0, q0, fma(q1, q1, fma(q2, q2, q3 * q3)));
      }
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (c >= 0 && c < k && s < best) { best = s; bi = c; }
    }
    if (have && l == 0 && bi != 0x7fffffff) {
      changed += (old_label != bi);
      labels[row] = bi;
      // the moved-rows map of the fast kernel has a zero for this row
      if (moved_bits != nullptr && count_changes && old_label != bi)
        atomicOr(&moved_bits[row >> 5], 1u << (unsigned int)(row & 31));
    }
  }
  if (count_changes) {
    changed = __reduce_add_sync(0xffffffffu, changed);
    if ((threadIdx.x & 31) == 0 && changed) atomicAdd(&st->changed, (unsigned long long)changed);
  }
}

}  // namespace km

// Host side of the tensor-core distance kernel: eligibility, the split centroid
// buffers, TMA tensor maps (encoded through the driver entry point, so the
// library has no link-time dependency on libcuda) and the launch.
#pragma once

#include "km_assign_tc.cuh"
#include "km_push.cuh"

namespace km {
namespace tc {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// rows x cols row-major matrix of fp32 (elem 4) or fp16 (elem 2), boxes of box_rows rows x
// 128 bytes, 128-byte swizzle
inline int make_map(CUtensorMap* map, const void* base, size_t rows, int cols, int box_rows, int elem) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) KM_FAIL(KM_ECUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t gstride[1] = {(cuuint64_t)cols * elem};
  cuuint32_t box[2] = {(cuuint32_t)(128 / elem), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1u, 1u};
  CUresult r = fn(map, elem == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                  const_cast<void*>(base), gdim, gstride, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) KM_FAIL(KM_ECUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
  return KM_OK;
}

struct Plan {
  __half* bhi = nullptr;   // [npad][64] upper halves of -2 c * sb
  __half* blo = nullptr;   // [npad][64] lower halves
  float* cn = nullptr;     // [npad] |c|^2 * sx * sb (+inf padding), [npad] max |c|^2
  float* xnorm = nullptr;  // [rows] |x|^2
  size_t xnorm_cap = 0;
  const float* xnorm_of = nullptr;
  size_t xnorm_rows = 0;
  int npad = 0, k = 0, d = 0;
  const float* x_base = nullptr;
  size_t x_rows = 0;
  float sx = 1.f, sb = 1.f;
  CUtensorMap tmX, tmBhi, tmBlo;
  bool ready = false;
  // the rows rounded once to fp16 (d = 64), and per row |x|^2 and the length of what the rounding left out
  __half* xsplit = nullptr;
  float2* xrowq = nullptr;
  size_t xsplit_cap = 0;
  const float* xsplit_of = nullptr;
  size_t xsplit_rows = 0;
  float xsplit_sx = 0.f;
  bool xsplit_failed = false;   // no memory for it: stay with the converting kernel
  CUtensorMap tmXh;

  void release() {
    km_free(bhi); km_free(blo); km_free(cn); km_free(xnorm); km_free(xsplit); km_free(xrowq);
    bhi = blo = nullptr;
    cn = xnorm = nullptr;
    xsplit = nullptr;
    xrowq = nullptr;
    xnorm_cap = xsplit_cap = 0;
    xnorm_of = xsplit_of = nullptr;
    ready = false;
  }
};

// Power-of-two scales that put x * sx and 2 c * sb below 2^14 (fp16 overflows at 65504):
// xmax bounds |x|, cbound bounds |c| (centroids are means of rows, or the caller's
// initial table).  Returns false when the magnitudes cannot be scaled into range.
inline bool pick_scales(double xmax, double cbound, float* sx, float* sb) {
  int ex = 0, ec = 0;
  if (xmax > 0) std::frexp(xmax, &ex);
  if (cbound > 0) std::frexp(cbound, &ec);
  const int px = 14 - ex, pb = 13 - ec;
  if (px < -100 || px > 100 || pb < -100 || pb > 100 || px + pb < -120 || px + pb > 120) return false;
  *sx = (float)std::ldexp(1.0, px);
  *sb = (float)std::ldexp(1.0, pb);
  return true;
}

inline bool shape_ok(int k, int d) { return (d == 32 || d == 64) && k > 16 && k <= kMaxNPad; }

// |x|^2 per row, once per attached matrix
inline int ensure_xnorm(Plan& pl, const float* X, size_t rows, int d, int num_sms, cudaStream_t stream) {
  if (pl.xnorm_of != X || pl.xnorm_rows != rows) {
    if (pl.xnorm_cap < rows) {
      km_free(pl.xnorm);
      pl.xnorm = nullptr;
      KM_CUDA(km_malloc(&pl.xnorm, rows * sizeof(float)));
      pl.xnorm_cap = rows;
    }
    rownorm_kernel<<<num_sms * 8, 256, 0, stream>>>(X, rows, d, pl.xnorm);
    KM_CUDA(cudaGetLastError());
    pl.xnorm_of = X;
    pl.xnorm_rows = rows;
  }
  return KM_OK;
}

// The fp16 copy of X for the kernel variant without converter warps (d = 64): made when the
// matrix, its size or the scale changed; costs one pass over X and half as much memory again.
inline bool presplit_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("H2O4GPU_KM_TC_PRESPLIT");
    return !(e && e[0] == '0');
  }();
  return on;
}
inline bool ensure_xsplit(Plan& pl, const float* X, size_t rows, int d, float sx, int num_sms, cudaStream_t stream,
                          bool allow_build) {
  if (d != 64 || !presplit_enabled() || pl.xsplit_failed) return false;
  if (pl.xsplit && pl.xsplit_of == X && pl.xsplit_rows == rows && pl.xsplit_sx == sx) return true;
  if (!allow_build) return false;   // a single pass (predict) does not pay for the split
  if (pl.xsplit_cap < rows) {
    km_free(pl.xsplit);
    km_free(pl.xrowq);
    pl.xsplit = nullptr;
    pl.xrowq = nullptr;
    pl.xsplit_cap = 0;
    const size_t row_bytes = 64 * sizeof(__half) + sizeof(float2);
    if (!km_room_for(rows * row_bytes) || km_malloc(&pl.xsplit, rows * 64 * sizeof(__half)) != cudaSuccess ||
        km_malloc(&pl.xrowq, rows * sizeof(float2)) != cudaSuccess) {
      cudaGetLastError();
      km_free(pl.xsplit);   // one without the other is of no use
      pl.xsplit = nullptr;
      pl.xrowq = nullptr;
      pl.xsplit_failed = true;
      return false;
    }
    pl.xsplit_cap = rows;
  }
  split_rows_kernel<<<num_sms * 8, 256, 0, stream>>>(X, rows, sx, pl.xsplit, pl.xrowq);
  if (cudaGetLastError() != cudaSuccess || make_map(&pl.tmXh, pl.xsplit, rows, 64, kBM, 2) != KM_OK) {
    pl.xsplit_failed = true;
    return false;
  }
  pl.xsplit_of = X;
  pl.xsplit_rows = rows;
  pl.xsplit_sx = sx;
  return true;
}

inline int setup(Plan& pl, const float* X, size_t rows, int k, int d, int num_sms, cudaStream_t stream) {
  const int npad = (k + 15) / 16 * 16;
  if (pl.ready && pl.k == k && pl.d == d && pl.x_base == X && pl.x_rows == rows) return KM_OK;
  if (!(pl.bhi && pl.k == k && pl.d == d)) {
    km_free(pl.bhi); km_free(pl.blo); km_free(pl.cn);
    pl.bhi = pl.blo = nullptr;
    pl.cn = nullptr;
    KM_CUDA(km_malloc(&pl.bhi, (size_t)npad * 64 * sizeof(__half)));
    KM_CUDA(km_malloc(&pl.blo, (size_t)npad * 64 * sizeof(__half)));
    KM_CUDA(km_malloc(&pl.cn, (size_t)(npad + 1) * sizeof(float)));
  }
  pl.npad = npad; pl.k = k; pl.d = d; pl.x_base = X; pl.x_rows = rows;
  KM_TRY(make_map(&pl.tmX, X, rows, d, kBM, 4));
  KM_TRY(make_map(&pl.tmBhi, pl.bhi, npad, 64, npad, 2));
  KM_TRY(make_map(&pl.tmBlo, pl.blo, npad, 64, npad, 2));
  pl.ready = true;
  return KM_OK;
}

// rule: centroids the table leaves out (none for distances, which are wanted for all)
inline int prep(Plan& pl, const float* C, const float* cnorm, const OutRule& rule, cudaStream_t stream) {
  KM_CUDA(cudaMemsetAsync(pl.cn + pl.npad, 0, sizeof(float), stream));
  prep_kernel<<<pl.npad, 64, 0, stream>>>(C, cnorm, pl.k, pl.d, pl.npad, pl.sb, pl.sx * pl.sb, pl.bhi, pl.blo, pl.cn,
                                         rule);
  KM_CUDA(cudaGetLastError());
  return KM_OK;
}

// A row goes to the exact pass when second - best <= split_tolerance(...) (km_assign_tc.cuh):
// kTolRel * (|x|^2 + max|c|^2) plus an absolute floor.  Error of the split product with
// y = x sx = xh + xl + ex, b = -2c sb = bh + bl + eb: the kernel forms xh.bh + xl.bh + xh.bl, so a
// score misses xl.bl + ex.b + y.eb per element.  While the low halves are normal fp16 numbers
// |ex| <= 2^-22 |y|, |eb| <= 2^-22 |b|, |xl.bl| <= 2^-22 |y||b|: 3 * 2^-22 sum|y||b|
// <= 3 * 2^-22 (|x|^2 + |c|^2) sx sb per score; with the fp32 accumulation of the 3 d / 16 partial
// sums that is below 2^-20.4 (|x|^2 + |c|^2), twice that for a difference: kTolRel = 2^-19.
// A low half below 2^-14 is an fp16 subnormal (quantum 2^-24): |ex|, |eb| <= 2^-25 absolute,
// which adds 2^-25 (|y|_1 + |b|_1) per score; tol_floor_of(d) = 2^-23 sqrt(d) bounds twice that
// for a difference through |v|_1 <= sqrt(d) |v|_2.
// The accumulation term grows with the row width: the tensor core adds every K = 16 slice into the fp32
// accumulator with truncation, a one-sided error per step that is proportional to the accumulator's
// magnitude.  Measured on the worst case for it (all coordinates near a common offset, so that
// |x.c| = |x||c| and the accumulator reaches |x|^2 + |c|^2), the largest error of a single score was
// (0.38 + d / 210) * 2^-19 (|x|^2 + |c|^2): 2^-19.5 at d = 64, 2^-18.4 at 256, 2^-17.1 at 784, 2^-15.6 at 2048
// - the constant is the split error above (two-sided), the slope the truncation - and with the flat 2^-19
// rows of 2048 columns were mislabelled (3 of 40,000, gaps up to 3e-4 relative; none seen up to 784
// columns).  For the difference of two nearly tied scores the split errors add (2 * 0.38); the truncation
// errors have the sign of their accumulators: equal signs cancel in part, opposite signs mean
// |acc_j| + |acc_l| = | |c_l|^2 - |c_j|^2 | <= max|c|^2, so their sum stays below the single-score
// figure.  tol_rel_of(d) = 2^-19 (0.8 + d / 200) keeps 5 % above 2^-19 (0.76 + d / 210).
constexpr float kTolRel = 1.9073486328125e-06f;
inline float tol_rel_of(int d) { return kTolRel * (0.8f + (float)d / 200.0f); }
inline float tol_floor_of(int d) { return 1.1920928955078125e-07f * std::sqrt((float)d); }

inline int launch(Plan& pl, int* labels, IterState* st, bool count_changes, unsigned int* amb_rows,
                  unsigned int* amb_seg, float tol_rel, int num_sms, cudaStream_t stream, unsigned int* moved_bits,
                  uint4* amb_near, bool allow_split_build, int* launches) {
  const size_t tiles = (pl.x_rows + kBM - 1) / kBM;
  if (tiles > 0x7fffffffULL / kBM) KM_FAIL(KM_EINVAL, "shard too large for the tensor-core kernel");
  const int grid = (int)std::min<size_t>(tiles, (size_t)num_sms);
  const unsigned int seg_cap = (unsigned int)amb_seg_rows(pl.x_rows, num_sms);
  const bool pre = ensure_xsplit(pl, pl.x_base, pl.x_rows, pl.d, pl.sx, num_sms, stream, allow_split_build);
  if (!pre) KM_TRY(ensure_xnorm(pl, pl.x_base, pl.x_rows, pl.d, num_sms, stream));
  auto go = [&](auto fn, const CUtensorMap& tmX, bool p) -> int {
    KM_CUDA(allow_smem(fn, smem_bytes(pl.d, pl.npad, p)));
    fn<<<grid, kThreads, smem_bytes(pl.d, pl.npad, p), stream>>>(
        tmX, pl.tmBhi, pl.tmBlo, pl.cn, pl.xnorm, pl.xrowq, labels, pl.x_rows, (int)tiles, pl.npad, st,
        count_changes ? 1 : 0, amb_rows, amb_seg, seg_cap, tol_rel, tol_floor_of(pl.d), pl.sx, pl.sx * pl.sb,
        count_changes ? moved_bits : nullptr, amb_near, pre ? 1 : 0, wait_limits().mbar_iters);
    ++*launches;
    return KM_OK;
  };
  if (pl.d == 32) {
    KM_TRY(go(assign_tc_kernel<32, false>, pl.tmX, false));
  } else {
    if (pre) KM_TRY(go(assign_tc_kernel<64, true>, pl.tmXh, true));
    KM_TRY(go(assign_tc_kernel<64, false>, pl.tmX, false));
  }
  KM_CUDA(cudaGetLastError());
  return KM_OK;
}

}  // namespace tc
}  // namespace km

#include "km_assign_tc_big.cuh"

namespace km {
namespace tcb {

struct BigPlan {
  __half* bhi = nullptr;
  __half* blo = nullptr;
  float* cn = nullptr;     // [kpad] scaled |c|^2, [kpad] max |c|^2, [kpad + 1] longest remainder of the upper halves
  float* eb = nullptr;     // per centroid: length of what its upper halves leave out
  int kpad = 0, k = 0, d = 0, dp = 0;
  const float* x_base = nullptr;
  size_t x_rows = 0;
  float sx = 1.f, sb = 1.f;
  CUtensorMap tmX, tmBhi, tmBlo;
  bool ready = false;
  void release() {
    km_free(bhi); km_free(blo); km_free(cn); km_free(eb);
    bhi = blo = nullptr;
    cn = eb = nullptr;
    ready = false;
  }
};

// float32, rows of at most 256 columns with 16-byte alignment (d % 4 == 0); the |c|^2 table of all
// centroids must fit shared memory.  The kernel is compiled for 32, 64, 128 and 256 columns; other
// widths run the next larger variant: the copy engine zero-fills the columns of an X tile that lie
// beyond d and the split centroid table is zero there too, so the products are unchanged.
inline bool big_shape_ok(int k, int d) { return d >= 32 && d <= 256 && d % 4 == 0 && k > 16 && k <= 6144; }
inline int big_variant(int d) { return d <= 32 ? 32 : (d <= 64 ? 64 : (d <= 128 ? 128 : 256)); }

// the operand table: upper and lower halves (float32) or upper halves only (float64)
inline int big_tables(BigPlan& pl, int k, int d, bool lower) {
  const int kpad = (k + kNT - 1) / kNT * kNT;
  const int dv = big_variant(d);
  const int dp = dv < 64 ? 64 : dv;
  if (pl.eb && pl.k == k && pl.d == d) return KM_OK;
  pl.release();
  KM_CUDA(km_malloc(&pl.bhi, (size_t)kpad * dp * sizeof(__half)));
  if (lower) KM_CUDA(km_malloc(&pl.blo, (size_t)kpad * dp * sizeof(__half)));
  KM_CUDA(km_malloc(&pl.cn, (size_t)(kpad + 2) * sizeof(float)));
  KM_CUDA(km_malloc(&pl.eb, (size_t)kpad * sizeof(float)));
  pl.kpad = kpad; pl.k = k; pl.d = d; pl.dp = dp;
  KM_TRY(tc::make_map(&pl.tmBhi, pl.bhi, kpad, dp, kNT, 2));
  if (lower) KM_TRY(tc::make_map(&pl.tmBlo, pl.blo, kpad, dp, kNT, 2));
  return KM_OK;
}

// ldx: row pitch of X in elements (d, or d rounded up to four for the padded copy of unaligned rows)
inline int big_setup(BigPlan& pl, const float* X, size_t rows, int k, int d, int ldx) {
  KM_TRY(big_tables(pl, k, d, true));
  if (pl.ready && pl.x_base == X && pl.x_rows == rows) return KM_OK;
  pl.x_base = X; pl.x_rows = rows;
  KM_TRY(tc::make_map(&pl.tmX, X, rows, ldx, kBM, 4));
  pl.ready = true;
  return KM_OK;
}

template <typename T>
inline int big_prep(BigPlan& pl, const T* C, const T* cnorm, const OutRule& rule, cudaStream_t stream) {
  KM_CUDA(cudaMemsetAsync(pl.cn + pl.kpad, 0, 2 * sizeof(float), stream));
  big_prep_kernel<T><<<pl.kpad, 256, 0, stream>>>(C, cnorm, pl.k, pl.d, pl.dp, pl.kpad, pl.sb, pl.sx * pl.sb, pl.bhi,
                                                  pl.blo, pl.cn, pl.eb, rule);
  KM_CUDA(cudaGetLastError());
  return KM_OK;
}

template <int D>
inline int big_launch_d(BigPlan& pl, const float* xnorm, int xnorm_pitch, int* labels, IterState* st, int count_changes,
                        unsigned int* amb_rows, float tol_rel, int grid, int tiles, cudaStream_t stream, int gate) {
  KM_CUDA(allow_smem(assign_tc_big_kernel<D>, big_smem_bytes<D>(pl.kpad)));
  assign_tc_big_kernel<D><<<grid, kBigThreads, big_smem_bytes<D>(pl.kpad), stream>>>(
      pl.tmX, pl.tmBhi, pl.tmBlo, pl.cn, xnorm, xnorm_pitch, labels, pl.x_rows, tiles, pl.kpad, st, count_changes,
      amb_rows, tol_rel, tc::tol_floor_of(pl.d), pl.sx, pl.sx * pl.sb, gate, wait_limits().mbar_iters);
  KM_CUDA(cudaGetLastError());
  return KM_OK;
}

// gate: the kernel returns at once unless the one-product kernel in front of it gave the pass up; xnorm_pitch: floats
// from one row's |x|^2 to the next
inline int big_launch(BigPlan& pl, const float* xnorm, int xnorm_pitch, int* labels, IterState* st, bool count_changes,
                      unsigned int* amb_rows, float tol_rel, int num_sms, cudaStream_t stream, bool gate) {
  const size_t tiles = (pl.x_rows + kBM - 1) / kBM;
  if (tiles > 0x7fffffffULL / kBM) KM_FAIL(KM_EINVAL, "shard too large for the tensor-core kernel");
  const int grid = (int)std::min<size_t>(tiles, (size_t)num_sms);
  const int cc = count_changes ? 1 : 0;
  const int dv = big_variant(pl.d);
  auto go = [&](auto fn) {
    return fn(pl, xnorm, xnorm_pitch, labels, st, cc, amb_rows, tol_rel, grid, (int)tiles, stream, gate ? 1 : 0);
  };
  return dv == 32 ? go(big_launch_d<32>) : dv == 64 ? go(big_launch_d<64>)
       : dv == 128 ? go(big_launch_d<128>) : go(big_launch_d<256>);
}

}  // namespace tcb
}  // namespace km

#include "km_assign_tc_half.cuh"

namespace km {
namespace tch {

// What the one-product kernel keeps per matrix (the rounded rows) and per fit (the list of open rows); the centroid
// table is that of the three-term kernel (tcb::BigPlan).
struct HalfPlan {
  __half* xh = nullptr;           // [rows][ldh]
  float2* rowq = nullptr;         // [rows] |x|^2, length of the rounding's remainder
  size_t xh_cap = 0, rowq_cap = 0;
  const void* of = nullptr;       // matrix the rounded rows belong to (null: none)
  size_t rows = 0;
  int ldh = 0;
  float sx = 0.f;
  CUtensorMap tmX;
  uint4* cand_near = nullptr;
  unsigned int cand_cap = 0;
  bool on = false;                // the current E-steps run on the rounded rows
  bool alone = false;             // ... with nothing queued behind them (a single pass over unaligned rows)

  // a quarter of the rows: settling an open row costs about twice its share of the pass that needs no list
  static size_t list_rows(size_t rows) { return std::max<size_t>(rows / 4, std::min<size_t>(rows, 4096)); }
  bool holds(size_t rows, int d) const {
    return xh_cap >= rows * (size_t)((d + 7) / 8 * 8) && rowq_cap >= rows && cand_cap >= list_rows(rows);
  }
  size_t bytes() const { return xh_cap * sizeof(__half) + rowq_cap * sizeof(float2) + cand_cap * sizeof(uint4); }

  void release() {
    km_free(xh); km_free(rowq); km_free(cand_near);
    xh = nullptr; rowq = nullptr; cand_near = nullptr;
    xh_cap = rowq_cap = 0;
    cand_cap = 0;
    of = nullptr;
    on = alone = false;
  }
};

template <typename P>
inline bool half_grow(P** p, size_t* cap, size_t need) {
  if (*cap >= need) return true;
  km_free(*p);
  *p = nullptr;
  *cap = 0;
  if (km_malloc(p, need * sizeof(P)) != cudaSuccess) { cudaGetLastError(); return false; }
  *cap = need;
  return true;
}

// Rounded rows of X (made when the matrix or the scale changed) and the candidate list.  False: no memory for
// them (none of it is held then), the caller stays with the kernels that read the rows as they are.
template <typename T>
inline bool half_rows(HalfPlan& pl, const T* X, size_t rows, int d, float sx, int num_sms, cudaStream_t stream,
                      int* launches) {
  const int ldh = (d + 7) / 8 * 8;
  const size_t cap = HalfPlan::list_rows(rows), elems = rows * (size_t)ldh;
  if (!pl.holds(rows, d)) {
    size_t have = pl.cand_cap;
    pl.of = nullptr;
    if (!km_room_for(elems * sizeof(__half) + rows * sizeof(float2) + cap * sizeof(uint4)) ||
        !half_grow(&pl.cand_near, &have, cap) || !half_grow(&pl.xh, &pl.xh_cap, elems) ||
        !half_grow(&pl.rowq, &pl.rowq_cap, rows)) {
      pl.release();
      return false;
    }
    pl.cand_cap = (unsigned int)have;
  }
  if (pl.of == X && pl.rows == rows && pl.sx == sx && pl.ldh == ldh) return true;
  pl.of = nullptr;
  int lpr = 1;
  while (lpr < 32 && lpr * 4 < ldh) lpr *= 2;
  if (d % 4 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0)
    half_rows_kernel<T, true><<<num_sms * 8, 256, 0, stream>>>(X, rows, d, ldh, lpr, sx, pl.xh, pl.rowq);
  else
    half_rows_kernel<T, false><<<num_sms * 8, 256, 0, stream>>>(X, rows, d, ldh, lpr, sx, pl.xh, pl.rowq);
  if (cudaGetLastError() != cudaSuccess || tc::make_map(&pl.tmX, pl.xh, rows, ldh, kBM, 2) != KM_OK) return false;
  ++*launches;
  pl.of = X;
  pl.rows = rows;
  pl.sx = sx;
  pl.ldh = ldh;
  return true;
}

template <int P>
inline int half_launch_p(HalfPlan& pl, tcb::BigPlan& tb, int* labels, IterState* st, bool count_changes, float tol_rel,
                         int num_sms, cudaStream_t stream, unsigned int* host_whole) {
  const size_t n_sub = (pl.rows + kBM - 1) / kBM;
  if (n_sub > 0x7fffffffULL / kBM) KM_FAIL(KM_EINVAL, "shard too large for the tensor-core kernel");
  const int grid = (int)std::min<size_t>(n_sub, (size_t)num_sms);
  const size_t smem = half_smem_bytes(tb.d, tb.kpad);
  KM_CUDA(allow_smem(assign_tc_half_kernel<P>, smem));
  // rows whose candidates cannot be told apart by chunk cost k / 32 times more in the exact pass; what takes over
  // costs three times the one-product pass for float32 rows and forty times as much for float64 ones
  const unsigned int all_limit = (unsigned int)std::max<size_t>(64, tb.blo ? pl.rows / 64 : pl.rows / 8);
  assign_tc_half_kernel<P><<<grid, kHalfThreads, smem, stream>>>(
      pl.tmX, tb.tmBhi, tb.cn, pl.rowq, labels, pl.rows, (int)n_sub, tb.kpad, (tb.d + 15) / 16, st,
      count_changes ? 1 : 0, pl.cand_near, pl.cand_cap, all_limit, tol_rel, tc::tol_floor_of(tb.d),
      tb.sx, tb.sx * tb.sb, wait_limits().mbar_iters, host_whole);
  KM_CUDA(cudaGetLastError());
  return KM_OK;
}

// host_whole (or null): pinned word that receives st->full_rows as the kernel leaves it
inline int half_launch(HalfPlan& pl, tcb::BigPlan& tb, int* labels, IterState* st, bool count_changes, float tol_rel,
                       int num_sms, cudaStream_t stream, unsigned int* host_whole) {
  switch (panels_of(tb.d)) {
    case 1: return half_launch_p<1>(pl, tb, labels, st, count_changes, tol_rel, num_sms, stream, host_whole);
    case 2: return half_launch_p<2>(pl, tb, labels, st, count_changes, tol_rel, num_sms, stream, host_whole);
    case 3: return half_launch_p<3>(pl, tb, labels, st, count_changes, tol_rel, num_sms, stream, host_whole);
    default: return half_launch_p<4>(pl, tb, labels, st, count_changes, tol_rel, num_sms, stream, host_whole);
  }
}

}  // namespace tch
}  // namespace km

#include "km_assign_tc_wide.cuh"

namespace km {
namespace tcw {

struct WidePlan {
  __half* bhi = nullptr;
  __half* blo = nullptr;
  float* cn = nullptr;
  int k = 0, d = 0, dp = 0, n_chunks = 0, stages = 0;
  const float* x_base = nullptr;
  size_t x_rows = 0;
  float sx = 1.f, sb = 1.f;
  CUtensorMap tmX, tmBhi, tmBlo;
  bool ready = false;
  void release() {
    km_free(bhi); km_free(blo); km_free(cn);
    bhi = blo = nullptr;
    cn = nullptr;
    ready = false;
  }
};

// Ring depth for d columns: four stages, or two when shared memory is short.  EVEN on purpose: chunks
// alternate between the two converter groups, so with an even depth a stage always serves the same
// group and every "stage full" barrier has one waiter that takes its phases in order.  With an odd
// depth the two groups would share a stage's barrier without being ordered against each other, and a
// one-bit phase parity cannot tell "the phase I wait for" from "the phase before the previous one":
// a group that ran ahead of a late copy took the stage early (a device fault at 2e6 rows x 784).
inline int wide_stages(int d) {
  const int n_chunks = (d + kChunk - 1) / kChunk;
  for (int s = 4; s >= 2; s -= 2)
    if (wide_smem_bytes(n_chunks, s) <= (size_t)227 * 1024) return s;
  return 0;
}
// float32, at most 16 centroids, rows of 128 or more columns (16-byte aligned rows: d % 4 == 0)
inline bool wide_shape_ok(int k, int d) { return k >= 1 && k <= kNPad && d >= 128 && d % 4 == 0 && wide_stages(d) > 0; }

inline int wide_setup(WidePlan& pl, const float* X, size_t rows, int k, int d, int ldx) {
  if (pl.ready && pl.k == k && pl.d == d && pl.x_base == X && pl.x_rows == rows) return KM_OK;
  const int n_chunks = (d + kChunk - 1) / kChunk;
  const int dp = n_chunks * kChunk;
  if (!(pl.bhi && pl.k == k && pl.d == d)) {
    pl.release();
    KM_CUDA(km_malloc(&pl.bhi, (size_t)kNPad * dp * sizeof(__half)));
    KM_CUDA(km_malloc(&pl.blo, (size_t)kNPad * dp * sizeof(__half)));
    KM_CUDA(km_malloc(&pl.cn, (size_t)(kNPad + 1) * sizeof(float)));
  }
  pl.k = k; pl.d = d; pl.dp = dp; pl.n_chunks = n_chunks; pl.stages = wide_stages(d);
  pl.x_base = X; pl.x_rows = rows;
  KM_TRY(tc::make_map(&pl.tmX, X, rows, ldx, kBM, 4));
  KM_TRY(tc::make_map(&pl.tmBhi, pl.bhi, kNPad, dp, kNPad, 2));
  KM_TRY(tc::make_map(&pl.tmBlo, pl.blo, kNPad, dp, kNPad, 2));
  pl.ready = true;
  return KM_OK;
}

inline int wide_prep(WidePlan& pl, const float* C, const float* cnorm, const OutRule& rule, cudaStream_t stream) {
  KM_CUDA(cudaMemsetAsync(pl.cn + kNPad, 0, sizeof(float), stream));
  tcb::big_prep_kernel<float><<<kNPad, 256, 0, stream>>>(C, cnorm, pl.k, pl.d, pl.dp, kNPad, pl.sb, pl.sx * pl.sb,
                                                         pl.bhi, pl.blo, pl.cn, nullptr, rule);
  KM_CUDA(cudaGetLastError());
  return KM_OK;
}

// labels of rows [row0, row0 + nrows) (row0 a multiple of 128), or - with `out` - their squared distances to
// the k centroids as a column-major block with leading dimension ld_out
inline int wide_launch(WidePlan& pl, const float* xnorm, int* labels, IterState* st, bool count_changes,
                       unsigned int* amb_rows, float tol_rel, int num_sms, cudaStream_t stream, size_t row0 = 0,
                       size_t nrows = 0, float* out = nullptr, size_t ld_out = 0) {
  if (nrows == 0) nrows = pl.x_rows - row0;
  const size_t tiles = (nrows + kBM - 1) / kBM;
  if ((pl.x_rows + kBM - 1) / kBM > 0x7fffffffULL / kBM) KM_FAIL(KM_EINVAL, "shard too large for the tensor-core kernel");
  const int grid = (int)std::min<size_t>(tiles, (size_t)num_sms);
  KM_CUDA(allow_smem(assign_tc_wide_kernel, wide_smem_bytes(pl.n_chunks, pl.stages)));
  assign_tc_wide_kernel<<<grid, kWThreads, wide_smem_bytes(pl.n_chunks, pl.stages), stream>>>(
      pl.tmX, pl.tmBhi, pl.tmBlo, pl.cn, xnorm, labels, std::min(pl.x_rows, row0 + nrows), (int)(row0 / kBM), (int)tiles,
      pl.n_chunks, pl.stages, pl.k, st, count_changes ? 1 : 0, amb_rows, tol_rel, tc::tol_floor_of(pl.d), pl.sx,
      pl.sx * pl.sb, wait_limits().mbar_iters, out, ld_out);
  KM_CUDA(cudaGetLastError());
  return KM_OK;
}

}  // namespace tcw
}  // namespace km

#include "km_assign_tc_stream.cuh"

namespace km {
namespace tcs {

struct StreamPlan {
  __half* bhi = nullptr;
  __half* blo = nullptr;
  float* cn = nullptr;
  int k = 0, d = 0, dp = 0, n_chunks = 0, npad = 0, n_pass = 0, kpad = 0;
  const float* x_base = nullptr;
  size_t x_rows = 0;
  float sx = 1.f, sb = 1.f;
  CUtensorMap tmX, tmBhi, tmBlo;
  bool ready = false;
  void release() {
    km_free(bhi); km_free(blo); km_free(cn);
    bhi = blo = nullptr;
    cn = nullptr;
    ready = false;
  }
};

// float32, more than 16 centroids, 16-byte aligned rows of 32 to 4096 columns.  Up to 128 centroids run
// with N = 128 and two accumulators, more with N = 256 (one pass per 256 centroids).
inline bool stream_shape_ok(int k, int d) { return k > 16 && k <= 6144 && d >= 32 && d <= 4096 && d % 4 == 0; }
inline int stream_npad(int k) { return k <= 128 ? 128 : 256; }

inline int stream_setup(StreamPlan& pl, const float* X, size_t rows, int k, int d, int ldx) {
  if (pl.ready && pl.k == k && pl.d == d && pl.x_base == X && pl.x_rows == rows) return KM_OK;
  const int n_chunks = (d + kSChunk - 1) / kSChunk;
  const int dp = n_chunks * kSChunk;
  const int npad = stream_npad(k);
  const int n_pass = (k + npad - 1) / npad;
  const int kpad = n_pass * npad;
  if (!(pl.bhi && pl.k == k && pl.d == d)) {
    pl.release();
    KM_CUDA(km_malloc(&pl.bhi, (size_t)kpad * dp * sizeof(__half)));
    KM_CUDA(km_malloc(&pl.blo, (size_t)kpad * dp * sizeof(__half)));
    KM_CUDA(km_malloc(&pl.cn, (size_t)(kpad + 1) * sizeof(float)));
  }
  pl.k = k; pl.d = d; pl.dp = dp; pl.n_chunks = n_chunks; pl.npad = npad; pl.n_pass = n_pass; pl.kpad = kpad;
  pl.x_base = X; pl.x_rows = rows;
  KM_TRY(tc::make_map(&pl.tmX, X, rows, ldx, kBM, 4));
  KM_TRY(tc::make_map(&pl.tmBhi, pl.bhi, kpad, dp, npad, 2));
  KM_TRY(tc::make_map(&pl.tmBlo, pl.blo, kpad, dp, npad, 2));
  pl.ready = true;
  return KM_OK;
}

inline int stream_prep(StreamPlan& pl, const float* C, const float* cnorm, const OutRule& rule, cudaStream_t stream) {
  KM_CUDA(cudaMemsetAsync(pl.cn + pl.kpad, 0, sizeof(float), stream));
  tcb::big_prep_kernel<float><<<pl.kpad, 256, 0, stream>>>(C, cnorm, pl.k, pl.d, pl.dp, pl.kpad, pl.sb, pl.sx * pl.sb,
                                                          pl.bhi, pl.blo, pl.cn, nullptr, rule);
  KM_CUDA(cudaGetLastError());
  return KM_OK;
}

// labels of rows [row0, row0 + nrows) (row0 a multiple of 128), or - with `out` - their squared distances to
// the k centroids as a column-major block with leading dimension ld_out
inline int stream_launch(StreamPlan& pl, const float* xnorm, int* labels, IterState* st, bool count_changes,
                         unsigned int* amb_rows, float tol_rel, int num_sms, cudaStream_t stream, size_t row0 = 0,
                         size_t nrows = 0, float* out = nullptr, size_t ld_out = 0) {
  if (nrows == 0) nrows = pl.x_rows - row0;
  const size_t tiles = (nrows + kBM - 1) / kBM;
  if ((pl.x_rows + kBM - 1) / kBM > 0x7fffffffULL / kBM) KM_FAIL(KM_EINVAL, "shard too large for the tensor-core kernel");
  const int grid = (int)std::min<size_t>(tiles, (size_t)num_sms);
  const size_t n_end = std::min(pl.x_rows, row0 + nrows);
  if (pl.npad == 128) {
    KM_CUDA(allow_smem(assign_tc_stream_kernel<128>, stream_smem_bytes<128>()));
    assign_tc_stream_kernel<128><<<grid, kSThreads, stream_smem_bytes<128>(), stream>>>(
        pl.tmX, pl.tmBhi, pl.tmBlo, pl.cn, xnorm, labels, n_end, (int)(row0 / kBM), (int)tiles, pl.n_chunks, pl.n_pass,
        pl.k, st, count_changes ? 1 : 0, amb_rows, tol_rel, tc::tol_floor_of(pl.d), pl.sx, pl.sx * pl.sb,
        wait_limits().mbar_iters, out, ld_out);
  } else {
    KM_CUDA(allow_smem(assign_tc_stream_kernel<256>, stream_smem_bytes<256>()));
    assign_tc_stream_kernel<256><<<grid, kSThreads, stream_smem_bytes<256>(), stream>>>(
        pl.tmX, pl.tmBhi, pl.tmBlo, pl.cn, xnorm, labels, n_end, (int)(row0 / kBM), (int)tiles, pl.n_chunks, pl.n_pass,
        pl.k, st, count_changes ? 1 : 0, amb_rows, tol_rel, tc::tol_floor_of(pl.d), pl.sx, pl.sx * pl.sb,
        wait_limits().mbar_iters, out, ld_out);
  }
  KM_CUDA(cudaGetLastError());
  return KM_OK;
}

}  // namespace tcs
}  // namespace km

// Labels of narrow rows (at most eight columns) for more than 16 centroids, float32 and float64.
//
// Replaces calculate_distances + relabel (src/gpu/kmeans/kmeans_labels.cu:115-244, kmeans_labels.h:360-392).
// The tile kernel pads a row to 16 columns: with three columns four fifths of its arithmetic are on zeros.  Here a
// thread keeps R rows in registers and walks the centroids, which all lanes read together from shared memory
// (d coordinates and |c|^2, padded to a vector load); the table passes through shared memory in pieces if it is
// large.  273,280 x 3 float64 rows, 64 centroids: 117 us with the tile kernel, 18 us now.  2e7 rows of them take
// 1.05 ms: the FP64 pipe at a third of its rate (d + 2 instructions per score) and issue slots half busy, the
// rest waits for the rows, which a thread loads before its first score.  The arithmetic is the tile kernel's - a
// chain of fused multiply-adds over the columns, then |c|^2 - 2 x.c, first minimum wins - so the labels are the
// same bit for bit.
#pragma once

#include "km_common.cuh"
#include "km_tiles.cuh"

namespace km {

constexpr int kNarrowThreads = 256;
constexpr int kNarrowPiece = 1024;    // centroids in shared memory at a time (at most 80 KB)
constexpr int kNarrowMaxD = 8;

// doubles / floats per centroid in shared memory: a whole number of 16-byte vectors
template <typename T> constexpr int narrow_pitch(int d) {
  return (d + 1 + (16 / (int)sizeof(T)) - 1) / (16 / (int)sizeof(T)) * (16 / (int)sizeof(T));
}

// rows per thread: independent chains that hide the latency, while enough CTAs remain to fill the GPU
template <typename T, int D, int R>
__global__ void __launch_bounds__(kNarrowThreads)
narrow_assign_kernel(const T* __restrict__ X, size_t n, const T* __restrict__ C, int k, const T* __restrict__ cnorm,
                     int* __restrict__ labels, IterState* st, const IterState* gate) {
  if (gate && !gate->full_rows) return;
  constexpr int PITCH = narrow_pitch<T>(D);
  constexpr int V = 16 / (int)sizeof(T);
  extern __shared__ __align__(16) unsigned char narrow_smem[];
  T* cs = reinterpret_cast<T*>(narrow_smem);
  const int tid = threadIdx.x;
  T x[R][D], best[R];
  int bi[R];
  const size_t base = (size_t)blockIdx.x * (kNarrowThreads * R) + tid;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const size_t row = base + (size_t)r * kNarrowThreads;
#pragma unroll
    for (int t = 0; t < D; ++t) x[r][t] = row < n ? X[row * D + t] : (T)0;
    best[r] = Inf<T>::v();
    bi[r] = 0;
  }
  for (int c0 = 0; c0 < k; c0 += kNarrowPiece) {
    const int kc = min(kNarrowPiece, k - c0);
    if (c0) __syncthreads();
    for (int i = tid; i < kc * D; i += kNarrowThreads) {
      const int c = i / D;
      cs[c * PITCH + (i - c * D)] = C[(size_t)c0 * D + i];
    }
    for (int c = tid; c < kc; c += kNarrowThreads) cs[c * PITCH + D] = cnorm[c0 + c];
    __syncthreads();
#pragma unroll 2
    for (int c = 0; c < kc; ++c) {
      T v[PITCH];
#pragma unroll
      for (int i = 0; i < PITCH / V; ++i) {
        T q[V];
        VecLoad<T, V>::ld(cs + c * PITCH + i * V, q);
#pragma unroll
        for (int j = 0; j < V; ++j) v[i * V + j] = q[j];
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        T dot = 0;
#pragma unroll
        for (int t = 0; t < D; ++t) dot = fma(x[r][t], v[t], dot);
        const T s = v[D] - (T)2 * dot;
        if (s < best[r]) { best[r] = s; bi[r] = c0 + c; }
      }
    }
  }
  unsigned int changed = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const size_t row = base + (size_t)r * kNarrowThreads;
    if (row < n) {
      changed += labels[row] != bi[r];
      labels[row] = bi[r];
    }
  }
  if (st) {
    changed = __reduce_add_sync(0xffffffffu, changed);
    if ((tid & 31) == 0 && changed) atomicAdd(&st->changed, (unsigned long long)changed);
  }
}

inline bool narrow_shape_ok(int k, int d) { return d >= 1 && d <= kNarrowMaxD && k > 16; }

template <typename T, int D>
inline int narrow_launch_d(const T* X, size_t n, const T* C, int k, const T* cnorm, int* labels, IterState* st,
                           const IterState* gate, int num_sms, cudaStream_t stream) {
  const size_t smem = (size_t)std::min(k, kNarrowPiece) * narrow_pitch<T>(D) * sizeof(T);
  auto go = [&](auto fn, int R) -> int {
    const size_t per = (size_t)kNarrowThreads * R, grid = (n + per - 1) / per;
    if (grid > 0x7fffffffULL) KM_FAIL(KM_EINVAL, "shard too large for one launch");
    KM_CUDA(allow_smem(fn, smem));
    fn<<<(unsigned)grid, kNarrowThreads, smem, stream>>>(X, n, C, k, cnorm, labels, st, gate);
    KM_CUDA(cudaGetLastError());
    return KM_OK;
  };
  // four rows per thread (two of float64) once that still leaves every SM four CTAs
  constexpr int R = sizeof(T) == 8 ? 2 : 4;
  if (n >= (size_t)num_sms * 4 * kNarrowThreads * R) return go(narrow_assign_kernel<T, D, R>, R);
  return go(narrow_assign_kernel<T, D, 1>, 1);
}

template <typename T>
inline int narrow_launch(const T* X, size_t n, int d, const T* C, int k, const T* cnorm, int* labels, IterState* st,
                         const IterState* gate, int num_sms, cudaStream_t stream) {
  switch (d) {
    case 1: return narrow_launch_d<T, 1>(X, n, C, k, cnorm, labels, st, gate, num_sms, stream);
    case 2: return narrow_launch_d<T, 2>(X, n, C, k, cnorm, labels, st, gate, num_sms, stream);
    case 3: return narrow_launch_d<T, 3>(X, n, C, k, cnorm, labels, st, gate, num_sms, stream);
    case 4: return narrow_launch_d<T, 4>(X, n, C, k, cnorm, labels, st, gate, num_sms, stream);
    case 5: return narrow_launch_d<T, 5>(X, n, C, k, cnorm, labels, st, gate, num_sms, stream);
    case 6: return narrow_launch_d<T, 6>(X, n, C, k, cnorm, labels, st, gate, num_sms, stream);
    case 7: return narrow_launch_d<T, 7>(X, n, C, k, cnorm, labels, st, gate, num_sms, stream);
    default: return narrow_launch_d<T, 8>(X, n, C, k, cnorm, labels, st, gate, num_sms, stream);
  }
}

}  // namespace km

// Sorted slices: a matrix of any pattern in slices of 32 rows whose lengths are
// nearly the same, for the persistent solves.
//
// The rows of a window (the rows that a CTA takes in one step: kSliceWindow or
// fewer) are ordered by length, then by their number of entries up to the
// diagonal, longest first, so that the rows of the learned factor and of its
// transpose have nearly the same lengths too; perm[slot] = row, and the columns
// are slots, so that the solve's vectors all live in slot order and only its ends
// see the permutation. Slice s holds slots 32 s .. 32 s + 31, lane = slot: entry k
// of a slice is at (base[s] + k) * 32 + lane, in the row's storage order, so that a
// row's products are added in that order; rows shorter than their slice end in
// entries of column -1, which are skipped. A geometric graph of mean degree 12
// (rows of 1-34 entries) pads by 6 % in A and 19 and 25 % in G and G^T in windows
// of 1024 rows (unsorted 52, 94 and 94 %; by length alone 3, 41 and 46 %). So
// that the warps of a CTA get the same work over its steps, every second step's
// slices run from the shortest to the longest, and each pair of steps starts with
// other warps (the pairs' starts spread over them).
//
// Against the tiles of k_crs (values and indices through shared memory): every
// load of the matrix is one run of 64 to 256 bytes per warp, straight to
// registers, a chunk ahead of its use, and no barrier in the product.
//
// What bounds it is the number of loads that 64 registers a thread keep in flight,
// then DRAM. us per iteration of the persistent solves on graphs, graph of kernels
// -> sorted slices (1,000,003 points: 149 MB in FP64, 23 us at the measured 6.54
// TB/s; 2,000,000 points learned: 400 MB, 61 us):
//   FP64     5,003: 19.6 -> 8.1   300,007: - -> 17   1,000,003: 71 -> 40   2M: 122 -> 80
//   mixed    5,003: 21.9 -> 8.6   300,007: - -> 15   1,000,003: - -> 31   2M: 85 -> 54
//   learned  5,003: 28.8 -> 15    300,007: - -> 31   1,000,003: - -> 65   2M: 161 -> 112
// Steps on the way (FP64 at 1M / learned at 2M): matrix through L1, 192 KB of
// resident vectors 52 / -; kept out of L1, 128-160 KB 47 / 144; loads past a
// slice's width predicated off instead of repeated 41.5 / 139; a chunk ahead 43 /
// 121; the pairs' starts spread 40 / 112. (4 entries at a time 44 / 142; FP64 with 8
// spills, 78.) Tried without gain: an L2 evict-last policy on part of the matrix, L2
// prefetch of the next slice or of the next product's first steps, 512-thread CTAs.
#pragma once

#include <cuda_bf16.h>

#include "device.cuh"

namespace cgx {

constexpr int kSliceWindow = 1024;
constexpr int kSliceMaxLen = 4095;  // entries of a row (12 bits of the sort key)

template <typename VT>
struct SliceView {
  const int *base;  // per slice, in units of 32 entries; one past the last too
  const int *col;   // slots; -1: no entry
  const VT *val;
  int N;
};

// --- build -------------------------------------------------------------------

// One CTA of `window` threads per window. perm, inv (row -> slot), and per slice
// the length of its longest row. *flag |= 1 for a row that is too long. grid: the
// CTAs of the solve, whose steps are `grid` windows each.
template <typename Rows>
__global__ void __launch_bounds__(kSliceWindow)
    k_slices_sort(int N, Rows A, int grid, int *__restrict__ perm, int *__restrict__ inv,
                  int *__restrict__ width, int *flag) {
  __shared__ unsigned long long key[kSliceWindow];
  const int T = blockDim.x, t = threadIdx.x, w0 = blockIdx.x * T, i = w0 + t;
  unsigned long long mine = 0;
  if (i < N) {
    const int j0 = A.begin(i), j1 = A.end(i);
    int len = j1 - j0, low = 0;
    if (len > kSliceMaxLen) {
      atomicOr(flag, 1);
      len = kSliceMaxLen;
    }
    for (int j = j0; j < j0 + len; j++) low += A.col(i, j) <= i;
    // Pairs of lengths, then the lower entries, rising and falling in turn: rows
    // that share a slice are near each other in both. (Ties in row order.)
    const int l2 = len / 2;
    mine = 1ull << 40 | (unsigned long long)l2 << 24 |
           (unsigned long long)((l2 & 1) ? low : 4095 - low) << 12 | (unsigned)(T - 1 - t);
  }
  key[t] = mine;
  // Bitonic sort, descending (T is a power of two).
  for (int k = 2; k <= T; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      __syncthreads();
      const int o = t ^ j;
      if (o > t) {
        const unsigned long long a = key[t], b = key[o];
        if (((t & k) == 0) == (a < b)) {
          key[t] = b;
          key[o] = a;
        }
      }
    }
  __syncthreads();
  mine = key[t];
  // Where the window's slices go (see above); the last, partial window's stay.
  const int S = T / 32, steps = ((int)gridDim.x + grid - 1) / grid, step = blockIdx.x / grid;
  const int rank = (step & 1) ? S - 1 - (t >> 5) : t >> 5;
  const int shift = (step >> 1) * S / ((steps + 1) >> 1);
  const int slot = w0 + T <= N ? w0 + (rank + shift) % S * 32 + (t & 31) : i;
  int len = 0;
  if (i < N) {
    const int row = w0 + T - 1 - (int)(mine & 4095u);
    perm[slot] = row;
    inv[row] = slot;
    len = A.end(row) - A.begin(row);
  }
  len = __reduce_max_sync(0xffffffffu, len);
  if ((t & 31) == 0 && i < N) width[slot >> 5] = len;
}

// The length of each slice's longest row under a given permutation.
template <typename Rows>
__global__ void __launch_bounds__(kThreads)
    k_slices_width(int N, Rows A, const int *__restrict__ perm, int *__restrict__ width) {
  const int lane = threadIdx.x & 31, slices = (N + 31) >> 5;
  for (int s = (blockIdx.x * kThreads + threadIdx.x) >> 5; s < slices;
       s += (gridDim.x * kThreads) >> 5) {
    const int slot = (s << 5) + lane, row = slot < N ? perm[slot] : 0;
    const int len =
        __reduce_max_sync(0xffffffffu, slot < N ? A.end(row) - A.begin(row) : 0);
    if (lane == 0) width[s] = len;
  }
}

// Columns and values, a warp per slice. base = the exclusive scan of width.
template <typename VT, typename Rows>
__global__ void __launch_bounds__(kThreads)
    k_slices_fill(int N, Rows A, const int *__restrict__ perm, const int *__restrict__ inv,
                  const int *__restrict__ base, int *__restrict__ col, VT *__restrict__ val) {
  const int lane = threadIdx.x & 31, slices = (N + 31) >> 5;
  for (int s = (blockIdx.x * kThreads + threadIdx.x) >> 5; s < slices;
       s += (gridDim.x * kThreads) >> 5) {
    const int slot = (s << 5) + lane, b = base[s], w = base[s + 1] - b;
    int row = 0, j0 = 0, len = 0;
    if (slot < N) {
      row = perm[slot];
      j0 = A.begin(row);
      len = A.end(row) - j0;
    }
    for (int k = 0; k < w; k++) {
      const size_t at = ((size_t)(b + k) << 5) + lane;
      col[at] = k < len ? inv[A.col(row, j0 + k)] : -1;
      val[at] = (VT)(k < len ? A.val(row, j0 + k) : decltype(A.val(row, 0))(0));
    }
  }
}

// --- the product's row -------------------------------------------------------

// Streamed once per product: kept out of L1, which the gathers need. Without `on`
// nothing is read (-1, 0): a predicate, where a condition in C++ would become a
// branch per load.
__device__ __forceinline__ int slice_load(const int *p, bool on) {
  int v;
  asm("{.reg .pred q; setp.ne.s32 q, %2, 0; mov.b32 %0, -1;\n"
      "@q ld.global.nc.L1::no_allocate.b32 %0, [%1];}"
      : "=r"(v)
      : "l"(p), "r"((int)on));
  return v;
}
__device__ __forceinline__ double slice_load(const double *p, bool on) {
  double v;
  asm("{.reg .pred q; setp.ne.s32 q, %2, 0; mov.f64 %0, 0d0000000000000000;\n"
      "@q ld.global.nc.L1::no_allocate.f64 %0, [%1];}"
      : "=d"(v)
      : "l"(p), "r"((int)on));
  return v;
}
__device__ __forceinline__ float slice_load(const float *p, bool on) {
  float v;
  asm("{.reg .pred q; setp.ne.s32 q, %2, 0; mov.f32 %0, 0f00000000;\n"
      "@q ld.global.nc.L1::no_allocate.f32 %0, [%1];}"
      : "=f"(v)
      : "l"(p), "r"((int)on));
  return v;
}
__device__ __forceinline__ float slice_load(const __nv_bfloat16 *p, bool on) {
  unsigned short v;
  asm("{.reg .pred q; setp.ne.s32 q, %2, 0; mov.u16 %0, 0;\n"
      "@q ld.global.nc.L1::no_allocate.u16 %0, [%1];}"
      : "=h"(v)
      : "l"(p), "r"((int)on));
  return __uint_as_float((unsigned)v << 16);
}
__device__ __forceinline__ double slice_mad(double s, double v, double x) { return madd(s, v, x); }
__device__ __forceinline__ float slice_mad(float s, float v, float x) { return fmaf(v, x, s); }

// Entries of a row that are loaded together (64 registers at 1024 threads).
constexpr int kSliceInFlight = 6, kSliceInFlight32 = 8;

// The products' rows over the slots of this CTA's steps: row(k, i, x_i, sum) for
// slot i of step k, x = xat(slot). The loads of the next U entries, of this slice
// or of the next one, are issued before the gathers of the current ones.
template <int TPB, int U, typename VT, typename XAt, typename Row>
__device__ __forceinline__ void slice_rows(const SliceView<VT> &A, int steps, XAt xat, Row row) {
  using Num = decltype(slice_load((const VT *)nullptr, true));
  const int lane = threadIdx.x & 31, slices = (A.N + 31) >> 5;
  const int stride = gridDim.x * (TPB / 32);
  int s = blockIdx.x * (TPB / 32) + (threadIdx.x >> 5), k = 0, k0 = 0;
  // Slice t of this warp: its first entry and width; none past the last.
  auto slice = [&](int t, int step, int &b, int &w) {
    b = w = 0;
    if (step < steps && t < slices) {
      b = __ldg(A.base + t);
      w = __ldg(A.base + t + 1) - b;
    }
  };
  auto load = [&](int b, int w, int j, int (&c)[U], Num (&v)[U]) {
    const int *__restrict__ col = A.col + (((size_t)b << 5) + lane);
    const VT *__restrict__ val = A.val + (((size_t)b << 5) + lane);
#pragma unroll
    for (int u = 0; u < U; u++) {
      c[u] = slice_load(col + ((j + u) << 5), j + u < w);
      v[u] = slice_load(val + ((j + u) << 5), j + u < w);
    }
  };
  int b, w, nb, nw, c[U];
  Num v[U], sum = 0;
  slice(s, 0, b, w);
  slice(s + stride, 1, nb, nw);
  load(b, w, 0, c, v);
  while (k < steps && s < slices) {
    const bool last = k0 + U >= w;
    const int j = last ? 0 : k0 + U;
    int cn[U], mb = 0, mw = 0;
    Num vn[U], x[U];
    load(last ? nb : b, last ? nw : w, j, cn, vn);
    if (last) slice(s + 2 * stride, k + 2, mb, mw);
#pragma unroll
    for (int u = 0; u < U; u++) x[u] = xat(max(c[u], 0));
#pragma unroll
    for (int u = 0; u < U; u++)
      if (c[u] >= 0) sum = slice_mad(sum, v[u], x[u]);
    if (last) {
      const int i = (s << 5) + lane;
      if (i < A.N) row(k, i, xat(i), sum);
      sum = 0;
      k++;
      s += stride;
      b = nb;
      w = nw;
      nb = mb;
      nw = mw;
    }
    k0 = j;
#pragma unroll
    for (int u = 0; u < U; u++) {
      c[u] = cn[u];
      v[u] = vn[u];
    }
  }
}

}  // namespace cgx

// Sorted slices: a matrix of any pattern in slices of 32 rows whose lengths are
// nearly the same, for the persistent solves.
//
// The rows of a window (the rows that a CTA takes in one step: kSliceWindow or
// fewer) are ordered by length, then by their number of entries up to the
// diagonal, longest first; perm[slot] = row, and the columns are slots too, so
// that the solve's vectors all live in slot order and only its ends see the
// permutation. Slice s holds slots 32 s .. 32 s + 31, lane = slot: entry k of a
// slot is at (base[s] + k) * 32 + lane, in the row's storage order, so that a
// row's products are added in that order; rows shorter than their slice end in
// entries of column -1, which are skipped. Sorted, a slice pads a geometric
// graph's rows (1-34 entries) by 4 %, where rows in their own order pad by 50 %.
// Every second step's slices run from the shortest to the longest, which evens
// out the warps of a CTA.
//
// Against the tiles of k_crs (values and indices through shared memory): every
// load of the matrix is one run of 128 or 256 bytes per warp, straight to
// registers, eight entries in flight per thread, and no barrier in the product.
//
// What it measured in FP64 on a graph of 1,000,003 points (12.4M entries, 149 MB,
// 23 us at the measured 6.54 TB/s; us per iteration of the persistent solve): 71 as
// the graph of k_crs_warp and the vector kernels; 52.5 with the matrix through L1
// and 192 KB of resident vectors; 45 with the matrix kept out of L1 and 128 to 160
// KB of them (96 KB 46, 64 KB 46); 4 entries in flight 47; without the prefetch of
// the next slice 48. Without its gathers (a column as the vector's value) the
// iteration takes 39: the stream and three barriers. Tried without gain: an L2
// evict-last policy on a part of the matrix (30 / 50 / 70 %: 45 / 49 / 51), the
// next product's first steps fetched into L2 before the barriers (one step 45.7,
// two 47.9, five 55), 512-thread CTAs with 8 or 16 entries in flight (55).
#pragma once

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
    // Valid, length, lower entries; ties in row order.
    mine = 1ull << 40 | (unsigned long long)len << 24 | (unsigned long long)low << 12 |
           (unsigned)(T - 1 - t);
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
  const bool full = w0 + T <= N, turn = full && ((blockIdx.x / grid) & 1);
  const int slot = turn ? w0 + (T - 32 - (t & ~31)) + (t & 31) : i;
  int len = 0;
  if (i < N) {
    const int row = w0 + T - 1 - (int)(mine & 4095u);
    perm[slot] = row;
    inv[row] = slot;
    len = (int)(mine >> 24) & 4095;
  }
  len = __reduce_max_sync(0xffffffffu, len);
  if ((t & 31) == 0 && i < N) width[slot >> 5] = len;
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
      val[at] = k < len ? (VT)A.val(row, j0 + k) : (VT)0;
    }
  }
}

// --- the product's row -------------------------------------------------------

#ifndef SLD
#define SLD 0
#endif
// Streamed once per product: kept out of L1, which the gathers need.
__device__ __forceinline__ int slice_load(const int *p) {
  int v;
  asm("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double slice_load(const double *p) {
  double v;
  asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double slice_mad(double s, double v, double x) { return madd(s, v, x); }

// L2 prefetch of `bytes` from p, 128 bytes per lane and turn.
__device__ __forceinline__ void slice_prefetch(const void *p, int bytes) {
  for (int o = 128 * (threadIdx.x & 31); o < bytes; o += 128 * 32)
    asm volatile("prefetch.global.L2 [%0];" : : "l"((const char *)p + o));
}

constexpr int kSliceInFlight = 8;  // entries of a row in flight

// The products' rows over the slots of this CTA's steps: row(k, i, x_i, sum) for
// slot i of step k, x = xat(slot). U entries' loads are issued before the first
// use (past the slice's width they re-read its last entries and are left out);
// the next step's slice is fetched into L2 meanwhile.
template <int TPB, int U, typename VT, typename XAt, typename Row>
__device__ __forceinline__ void slice_rows(const SliceView<VT> &A, int steps, XAt xat, Row row) {
  const int lane = threadIdx.x & 31, slices = (A.N + 31) >> 5;
  const int stride = gridDim.x * (TPB / 32);
  int s = blockIdx.x * (TPB / 32) + (threadIdx.x >> 5), b = 0, e = 0;
  if (s < slices) {
    b = __ldg(A.base + s);
    e = __ldg(A.base + s + 1);
  }
  for (int k = 0; k < steps && s < slices; k++, s += stride) {
    int nb = 0, ne = 0;
    if (k + 1 < steps && s + stride < slices) {
      nb = __ldg(A.base + s + stride);
      ne = __ldg(A.base + s + stride + 1);
    }
    const int i = (s << 5) + lane, w = e - b;
    const int *__restrict__ col = A.col + (((size_t)b << 5) + lane);
    const VT *__restrict__ val = A.val + (((size_t)b << 5) + lane);
    const auto xi = xat(min(i, A.N - 1));
    VT sum = 0;
    for (int k0 = 0; k0 < w; k0 += U) {
      int c[U];
      VT v[U], x[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int o = min(k0 + u, w - 1) << 5;
        c[u] = slice_load(col + o);
        v[u] = slice_load(val + o);
      }
      if (k0 == 0) {
        slice_prefetch(A.col + ((size_t)nb << 5), (ne - nb) * 32 * (int)sizeof(int));
        slice_prefetch(A.val + ((size_t)nb << 5), (ne - nb) * 32 * (int)sizeof(VT));
      }
#pragma unroll
      for (int u = 0; u < U; u++) x[u] = xat(max(c[u], 0));
#pragma unroll
      for (int u = 0; u < U; u++)
        if (k0 + u < w && c[u] >= 0) sum = slice_mad(sum, v[u], x[u]);
    }
    if (i < A.N) row(k, i, xi, sum);
    b = nb;
    e = ne;
  }
}

}  // namespace cgx

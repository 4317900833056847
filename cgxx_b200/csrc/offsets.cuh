// Values stored by offset: U + k * ld is an array over the rows with the entries
// on diagonal d[k]. FP64 for the plain solves (solve64.cuh), FP32 for the inner
// solves of matrices with more offsets than the row-major band holds
// (persist.cuh).
#pragma once

#include "band.cuh"

namespace cgx {

constexpr int kBand64MaxHalf = 14;  // stored offsets of a symmetric matrix
constexpr int kBand64MaxK = 27;     // stored offsets of any other

// The stored offsets, ascending, and the values by offset: U + k * ld, row
// i's entry A(i, i + d[k]), zero where row i has none. SYM: d[0] = 0 and the
// upper offsets. Padding slots have offset 0 and value 0.
template <int K, bool SYM, typename VT = double>
struct Band64View {
  const VT *U;
  size_t ld;
  int N;
  int d[K];
};

struct Band64Offsets {
  int K;
  int d[kBand64MaxK];
};

// --- build -------------------------------------------------------------------

__device__ __forceinline__ int band64_slot(const Band64Offsets &o, int d) {
  for (int k = 0; k < o.K; k++)
    if (o.d[k] == d) return k;
  return -1;
}

// U_k[i] = A(i, i + d_k); for SYM only the diagonal and above, and counts[0]
// += entries above the diagonal. *flag |= 2 for an offset outside the set or a
// row whose columns do not ascend.
template <bool SYM, typename VT, typename Rows>
__global__ void __launch_bounds__(kThreads)
    k_band64_fill(int N, Rows A, Band64Offsets o, VT *__restrict__ U, size_t ld,
                  unsigned long long *counts, int *flag) {
  unsigned long long upper = 0;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < N; i += gridDim.x * kThreads) {
    int last = -1;
    const int j1 = A.end(i);
    for (int j = A.begin(i); j < j1; j++) {
      const int c = A.col(i, j), d = c - i;
      if (c <= last) atomicOr(flag, 2);
      last = c;
      if (SYM && d < 0) continue;
      const int k = band64_slot(o, d);
      if (k < 0) {
        atomicOr(flag, 2);
        continue;
      }
      U[k * ld + i] = (VT)A.val(i, j);
      upper += d > 0;
    }
  }
  for (int s = 16; s > 0; s >>= 1) upper += __shfl_xor_sync(0xffffffffu, upper, s);
  if ((threadIdx.x & 31) == 0 && upper) atomicAdd(&counts[0], upper);
}

// Every lower entry must equal the upper entry of its mirror row bit for bit
// in value (a NaN fails). counts[1] += lower entries; with as many upper ones
// and no column twice in a row the pairing is one to one.
template <typename VT, typename Rows>
__global__ void __launch_bounds__(kThreads)
    k_band64_check(int N, Rows A, Band64Offsets o, const VT *__restrict__ U, size_t ld,
                   unsigned long long *counts, int *flag) {
  unsigned long long lower = 0;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < N; i += gridDim.x * kThreads) {
    const int j1 = A.end(i);
    for (int j = A.begin(i); j < j1; j++) {
      const int c = A.col(i, j), d = i - c;
      if (d <= 0) continue;
      const int k = band64_slot(o, d);
      if (k < 0 || U[k * ld + c] != (VT)A.val(i, j)) {
        atomicOr(flag, 4);
        continue;
      }
      lower++;
    }
  }
  for (int s = 16; s > 0; s >>= 1) lower += __shfl_xor_sync(0xffffffffu, lower, s);
  if ((threadIdx.x & 31) == 0 && lower) atomicAdd(&counts[1], lower);
}

}  // namespace cgx

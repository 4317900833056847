// Grid-wide sum that is also the barrier between two phases of a cooperative
// launch: every CTA contributes up to two doubles, and all leave with scalars
// computed from the grid's totals, which are added in one fixed order.
//
// What bounds it is latency: the release of the CTA's stores and its arrival
// (about 0.5 us), the poll that sees the last arrival (0.5 us), the loads of
// the partial sums (0.35 us), and the sums inside the CTA (0.25 us at 256
// threads, 0.4 us at 1024). So one warp does everything between the two CTA
// barriers: it forms the CTA's partial, arrives, polls, loads the partials
// (one round trip), sums them and computes the scalars (a division by every
// warp of a wide CTA costs as much as the partials' round trip). Two sums
// share their shuffles (warp_sum2). Measured back to back, 148 CTAs, one
// store per thread before each: 1.98 / 2.03 us for one / two sums at 256
// threads and 2.16 / 2.24 us at 1024; every thread summing the partials
// of each sum after a counter barrier takes 2.16 / 2.89 and 2.29 / 3.16 us (296
// CTAs of 1024 threads 3.05 / 3.92 us).
// Tried: the partial itself as the arrival, polled by every CTA (3.5-4.5 us at
// 148 CTAs: the polls of all slots queue in L2, also with the slots in up to
// eight copies), and one CTA that collects the slots and answers into a
// mailbox per CTA (3.1-4.0 us).
//
// Every wait on a grid is bounded (kSyncPolls polls); a CTA that gives up reports
// false and its kernel leaves the loop, sets kErrGridSync and returns.
#pragma once

#include "device.cuh"

namespace cgx {

constexpr unsigned kSyncPolls = 1u << 24;
enum : int { kErrGridSync = 4 };  // CgState::error: a grid barrier gave up

constexpr int kRedCtas = 320;  // most CTAs of a launch
constexpr int kRedVals = 2;
// Global memory of one launch: the arrival counter (zeroed by the host before
// the launch), then two sets of partial sums. A set is written again two
// rounds later, by when every CTA has arrived at the round between and so has
// read it.
// The counter and each flag of wait_below have a 128-byte line of their own.
constexpr int kRedLine = 16;  // unsigned long longs
struct RedMem {
  unsigned long long count;
  unsigned long long pad[kRedLine - 1];
  unsigned long long flags[kRedCtas * kRedLine];
  double part[2][kRedVals][kRedCtas];
};
constexpr size_t kRedZeroBytes = sizeof(unsigned long long) * kRedLine * (1 + kRedCtas);

__device__ __forceinline__ unsigned long long ld_acquire_u64(
    const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ double warp_sum_all(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums of a and b over the warp with the shuffles of little more than one: a's
// in lanes 0-15, b's in lanes 16-31.
__device__ __forceinline__ double warp_sum2(double a, double b) {
  const bool low = (threadIdx.x & 31) < 16;
  double mine = low ? a : b;
  const double other = low ? b : a;
  mine += __shfl_xor_sync(0xffffffffu, other, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  return mine;
}

template <int NV>
__device__ __forceinline__ void warp_sums(double (&v)[NV]) {
  if constexpr (NV == 2) {
    const double s = warp_sum2(v[0], v[1]);
    v[0] = __shfl_sync(0xffffffffu, s, 0);
    v[1] = __shfl_sync(0xffffffffu, s, 16);
  } else {
    v[0] = warp_sum_all(v[0]);
  }
}

// Barrier over the grid. fin(s, sc) runs in one thread of every CTA with the
// grid's sums s (NV > 0) and fills sc, a shared array that every thread may
// read after the call. Returns false when the wait gave up. Called by all
// threads of all CTAs; `round` is each thread's own count of calls, from 0.
template <int TPB, int NV, typename Fin>
__device__ __forceinline__ bool grid_sum(RedMem *m, unsigned &round,
                                         const double (&v)[NV > 0 ? NV : 1], double *sc,
                                         Fin fin, unsigned polls = kSyncPolls) {
  constexpr int NS = NV > 0 ? NV : 1, kWarpsT = TPB / 32, kPer = kRedCtas / 32;
  static_assert(NV <= kRedVals && TPB % 32 == 0 && TPB <= 1024, "grid_sum");
  __shared__ double sh[NS][kWarpsT];
  __shared__ int gave_up;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int G = (int)gridDim.x;
  double(*part)[kRedCtas] = m->part[round & 1];
  round++;
  if constexpr (NV == 2) {
    const double s = warp_sum2(v[0], v[1]);
    if ((lane & 15) == 0) sh[lane >> 4][w] = s;
  } else if constexpr (NV == 1) {
    const double s = warp_sum_all(v[0]);
    if (lane == 0) sh[0][w] = s;
  }
  __syncthreads();
  if (w == 0) {
    double s[NS];
    bool ok = true;
    if constexpr (NV > 0) {
#pragma unroll
      for (int a = 0; a < NS; a++) s[a] = lane < kWarpsT ? sh[a][lane] : 0.0;
      warp_sums<NS>(s);
    }
    if (G > 1) {
      if (lane == 0) {
        if constexpr (NV > 0) {
#pragma unroll
          for (int a = 0; a < NS; a++) __stcg(&part[a][blockIdx.x], s[a]);
        }
        // After the CTA barrier the add releases every thread's writes.
        asm volatile("red.release.gpu.global.add.u64 [%0], 1;" : : "l"(&m->count) : "memory");
        const unsigned long long target = (unsigned long long)round * G;
        unsigned i = 0;
        while (ld_acquire_u64(&m->count) < target && ++i < polls) __nanosleep(32);
        ok = i < polls;
      }
      __syncwarp();
      if constexpr (NV > 0) {
        double x[NS][kPer];
#pragma unroll
        for (int k = 0; k < kPer; k++) {
          const int j = lane + 32 * k;
#pragma unroll
          for (int a = 0; a < NS; a++) x[a][k] = j < G ? __ldcg(&part[a][j]) : 0.0;
        }
#pragma unroll
        for (int a = 0; a < NS; a++) {
          s[a] = 0.0;
#pragma unroll
          for (int k = 0; k < kPer; k++) s[a] += x[a][k];
        }
        warp_sums<NS>(s);
      }
    }
    if (lane == 0) {
      fin(s, sc);
      gave_up = !ok;
    }
  }
  __syncthreads();
  return !gave_up;
}

// The same for a launch that is one thread-block cluster (at most kClusterCtas
// CTAs): the partials go straight into every CTA's shared memory, and the
// cluster's hardware barrier, which needs no polls, makes them visible. It has no
// limit, but always ends, as the CTAs of a cluster run together and take the same
// decisions. A CTA's shared memory may be written only while it runs: every
// kernel calls cluster_sync before its first cluster_sum (the CTAs are scheduled
// together, but one without rows would store before a later one has started) and
// before a CTA returns (another may still write to it). A fused iteration on 64^2
// rows, two sums, takes 3.0 us with it and 4.8 on the grid.
constexpr int kClusterCtas = 16;
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void store_in_cta(double *p, int cta, double v) {
  unsigned at = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(at) : "r"(cta));
  asm volatile("st.shared::cluster.f64 [%0], %1;" : : "r"(at), "d"(v) : "memory");
}
template <int TPB, int NV, typename Fin>
__device__ __forceinline__ bool cluster_sum(unsigned &round, const double (&v)[NV], double *sc,
                                            Fin fin) {
  constexpr int kWarpsT = TPB / 32;
  static_assert(NV >= 1 && NV <= 2 && TPB % 32 == 0 && TPB <= 1024, "cluster_sum");
  __shared__ double sh[NV][kWarpsT];
  // Two sets in turn: a set is written again two rounds later, by when every CTA
  // has passed the barrier between and so has read it.
  __shared__ double part[2][NV][kClusterCtas];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, G = (int)gridDim.x;
  double(*mine)[kClusterCtas] = part[round & 1];
  round++;
  if constexpr (NV == 2) {
    const double s = warp_sum2(v[0], v[1]);
    if ((lane & 15) == 0) sh[lane >> 4][w] = s;
  } else {
    const double s = warp_sum_all(v[0]);
    if (lane == 0) sh[0][w] = s;
  }
  __syncthreads();
  double s[NV];
  if (w == 0) {
#pragma unroll
    for (int a = 0; a < NV; a++) s[a] = lane < kWarpsT ? sh[a][lane] : 0.0;
    warp_sums<NV>(s);
    if (lane < G) {
#pragma unroll
      for (int a = 0; a < NV; a++) store_in_cta(&mine[a][blockIdx.x], lane, s[a]);
    }
    __syncwarp();
  }
  cluster_sync();
  if (w == 0) {
#pragma unroll
    for (int a = 0; a < NV; a++) s[a] = lane < G ? mine[a][lane] : 0.0;
    warp_sums<NV>(s);
    if (lane == 0) fin(s, sc);
  }
  __syncthreads();
  return true;
}

template <int TPB>
__device__ __forceinline__ bool grid_barrier(RedMem *m, unsigned &round,
                                             unsigned polls = kSyncPolls) {
  const double none[1] = {0.0};
  return grid_sum<TPB, 0>(m, round, none, (double *)nullptr,
                          [](const double (&)[1], double *) {}, polls);
}

// A launch's sums and barriers: over one cluster, or over a cooperative grid.
template <bool CLUSTER, int TPB, int NV, typename Fin>
__device__ __forceinline__ bool sum_over(RedMem *m, unsigned &round, const double (&v)[NV],
                                         double *sc, Fin fin) {
  if constexpr (CLUSTER)
    return cluster_sum<TPB, NV>(round, v, sc, fin);
  else
    return grid_sum<TPB, NV>(m, round, v, sc, fin);
}
template <bool CLUSTER, int TPB>
__device__ __forceinline__ bool sync_over(RedMem *m, unsigned &round) {
  if constexpr (CLUSTER) {
    cluster_sync();
    return true;
  } else {
    return grid_barrier<TPB>(m, round);
  }
}

// Waits for the CTAs before this one only: CTA b publishes `round` in its flag
// and waits until the flags of CTAs b - 1, ..., b - n have reached it (n
// at most the CTA's width, CTAs below 0 skipped), so that this CTA sees what
// those wrote before. The host zeroes the flags before the launch.
template <int TPB>
__device__ __forceinline__ bool wait_below(unsigned long long *flags, int n,
                                           unsigned long long round,
                                           unsigned polls = kSyncPolls) {
  __shared__ int gave_up;
  __syncthreads();
  if (threadIdx.x == 0) {
    gave_up = 0;
    asm volatile("st.release.gpu.global.u64 [%0], %1;"
                 :
                 : "l"(flags + blockIdx.x * kRedLine), "l"(round)
                 : "memory");
  }
  __syncthreads();
  const int b = (int)blockIdx.x - 1 - (int)threadIdx.x;
  if ((int)threadIdx.x < n && b >= 0) {
    unsigned i = 0;
    while (ld_acquire_u64(flags + b * kRedLine) < round && ++i < polls) __nanosleep(32);
    if (i >= polls) gave_up = 1;
  }
  __syncthreads();
  return !gave_up;
}

}  // namespace cgx

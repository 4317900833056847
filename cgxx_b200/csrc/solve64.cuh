// Persistent FP64 solves.
//
// A whole plain FP64 PCG loop is one cooperative launch: on A by offset when its
// rows are sorted and its entries lie on few diagonals (structured-grid stencils),
// else on A in sorted slices (slices.cuh). What this buys against the graph of
// k_crs, k_pcg_update and k_pcg_direction:
//  - bytes (by offset): the CRS product reads 12 bytes per nonzero (84 per row of the
//    7-point matrix). The values are stored by offset (U_k is an array over
//    the rows) without indices: 8 bytes per offset and row, and if A is
//    symmetric, only the diagonal and the upper offsets (32 bytes per row); a
//    lower value is then the upper value of an earlier row, U_k[i - d_k],
//    which L1 or L2 still holds;
//  - the vectors that only their own row's thread touches (r, x, C, q) stay
//    in shared memory for the whole solve, as many rows of them as fit
//    (28 MB over 148 SMs: 3.5M rows of one vector);
//  - launches: no kernel boundaries, no while node; the loop's scalars come
//    with the barriers (gridred.cuh).
//
// Stored by offset, every load of a warp, the shifted lower ones included, is
// one run of 256 bytes. (Row-major rows, which the FP32 band uses, would
// spread the lower loads over 32-byte sectors: 32 bytes fetched from L2 for
// each 8 used.)
//
// The arithmetic is the graph path's: a row's products are added in ascending
// column order, each product and each sum rounded on its own; entries that a
// row does not have are skipped. Only the order of the dot products' sums
// differs.
//
// Two forms:
//   split  A  q = A p                            | <p,q> -> a
//          B  r -= a q                           | <r,r>, <r,Cr> -> test, b
//          E  x += a p, p = C r + b p            |
//   fused  A  p = z + b p_old, x += a_old p_old, q = A p | <p,q> -> a
//          B  r -= a q, z = C r                          | <r,r>, <r,z> -> test, b
// The fused form saves a barrier and forms p at every neighbour it reads from
// z and the last p (two arrays of p in turn); it is for the systems whose
// barriers cost more than those reads.
//
// What bounds it: up to 64^3 the barriers (2.0-2.5 us each, gridred.cuh); at
// 160^3 DRAM (104 bytes per row and iteration, 426 MB, of which DRAM carries 398:
// 77 us against 61 at the measured 6.54 TB/s). us per iteration, graph ->
// persistent: 64^2 5-point 17.5 -> 4.6, 257^2 19.3 -> 5.5, 97x64x83 7-point
// (ELL) 26.6 -> 11.2, 128^3 68.6 -> 36.4, 160^3 138 -> 77, 27-point 96^3 80 ->
// 43.5.
#pragma once

#include "band.cuh"
#include "gridred.cuh"
#include "offsets.cuh"
#include "slices.cuh"

namespace cgx {

// --- the product's row -------------------------------------------------------

// sum + v x rounded twice, skipped where the row has no such entry (v = 0),
// so that a value of x the row does not refer to cannot reach it.
__device__ __forceinline__ double band64_add(double sum, double v, double x) {
  return (__double_as_longlong(v) << 1) != 0 ? madd(sum, v, x) : sum;
}

// Row i of A times a vector whose element j is xat(j), in ascending column
// order. The loads of a group of slots are issued before its sums; up to 7
// slots the whole row is one group (one round trip).
template <int K, bool SYM, typename XAt>
__device__ __forceinline__ double band64_row(const Band64View<K, SYM> &B, int i, XAt xat) {
  const double *__restrict__ U = B.U;
  const unsigned nmax = (unsigned)(B.N - 1);
  double sum = 0.0;
  // SYM: slot s of the row is the lower offset K - 1 - s for s < K - 1, else
  // the stored offset s - (K - 1).
  constexpr int kSlots = SYM ? 2 * K - 1 : K, G = 7;
#pragma unroll
  for (int s0 = 0; s0 < kSlots; s0 += G) {
    double v[G], x[G];
#pragma unroll
    for (int g = 0; g < G; g++) {
      const int s = s0 + g;
      if (s >= kSlots) continue;
      if (SYM && s < K - 1) {
        const int k = K - 1 - s, j = i - B.d[k], jc = max(j, 0);
        v[g] = __ldg(U + k * B.ld + jc);
        x[g] = xat(jc);
        v[g] = j < 0 ? 0.0 : v[g];
      } else {
        const int k = SYM ? s - (K - 1) : s;
        v[g] = __ldg(U + k * B.ld + i);
        // A column outside [0, N) belongs to a value 0: any element does.
        x[g] = xat((int)min((unsigned)(i + B.d[k]), nmax));
      }
    }
#pragma unroll
    for (int g = 0; g < G; g++)
      if (s0 + g < kSlots) sum = band64_add(sum, v[g], x[g]);
  }
  return sum;
}

// L2 prefetch of the rows that a thread reads in its next step: one lane per
// 128-byte line of each array.
template <int K, bool SYM>
__device__ __forceinline__ void band64_prefetch(const Band64View<K, SYM> &B, int i, int stride) {
  const long long j = (long long)i + stride;
  if ((threadIdx.x & 15) == 0 && j < B.N) {
#pragma unroll
    for (int k = 0; k < K; k++)
      asm volatile("prefetch.global.L2 [%0];" : : "l"(B.U + k * B.ld + j));
  }
}

// --- the solve ---------------------------------------------------------------

// The matrix of a solve. kPerm: the solve's rows are slots of the sorted slices,
// and the vectors are brought into their order and back.
template <int K, bool SYM, bool PF>
struct BandMat {
  static constexpr bool kPerm = false;
  Band64View<K, SYM> B;
  __device__ int n() const { return B.N; }
  __device__ int from(int i) const { return i; }
  __device__ void prefetch(int i, int stride) const {
    if (PF) band64_prefetch(B, i, stride);
  }
  template <typename XAt>
  __device__ double row(int i, XAt xat) const {
    return band64_row(B, i, xat);
  }
};
struct SliceMat {
  static constexpr bool kPerm = true;
  SliceView<double> S;
  const int *perm;
  __device__ int n() const { return S.N; }
  __device__ int from(int i) const { return __ldg(perm + i); }
};

struct Solve64Args {
  double *x, *r, *q;
  const double *C;  // NULL: no preconditioner (z = r)
  double *p;        // the direction; fused: in turn with p2
  double *p2, *z;   // fused only
  // kPerm: the same vectors in the matrix's own row order, read at the start and
  // written at the end (x, r, q, C and p above are then in slot order).
  double *xo, *ro, *qo, *po;
  const double *Co;
  RedMem *red;              // barrier state, its counter 0 at launch
  int steps;                // rows per thread
  int nr, nx, nc, nq;       // steps of r, x, C, q held in shared memory
};

// Where row i, step k of a vector lives: the first n steps in shared memory
// (sm: TPB elements per step), the rest in the global array.
template <int TPB>
__device__ __forceinline__ double *vec_at(double *sm, int n, double *g, int k, int i) {
  return k < n ? sm + (k * TPB + (int)threadIdx.x) : g + i;
}

template <typename Mat, bool FUSED, bool CLUSTER, int TPB>
__global__ void __launch_bounds__(TPB, 1) k_solve64(Mat A, Solve64Args a, CgState *st) {
  constexpr bool PERM = Mat::kPerm;
  static_assert(!(PERM && FUSED), "the fused form is the band's");
  extern __shared__ __align__(16) double sm[];
  __shared__ double sc[8];  // scalars of the last grid sum
  double *const sr = sm;
  double *const sx = sr + (size_t)a.nr * TPB;
  double *const scd = sx + (size_t)a.nx * TPB;
  double *const sq = scd + (size_t)a.nc * TPB;
  const int N = A.n(), steps = a.steps;
  const int i0 = blockIdx.x * TPB + threadIdx.x, stride = gridDim.x * TPB;
  const double nrm0 = st->nrm0, tol = st->tol;
  const int maxit = st->max_iter;
  double rho = st->rho, rho_old = 0.0, alpha = 0.0, beta = 0.0;
  int it = 0, conv = 0;
  unsigned round = 0;
  bool ok = true;

  for (int k = 0, i = i0; k < steps && i < N; k++, i += stride) {
    if constexpr (PERM) {
      const int j = A.from(i);
      *vec_at<TPB>(sr, a.nr, a.r, k, i) = a.ro[j];
      *vec_at<TPB>(sx, a.nx, a.x, k, i) = a.xo[j];
      if (a.C) *vec_at<TPB>(scd, a.nc, const_cast<double *>(a.C), k, i) = a.Co[j];
      a.p[i] = a.po[j];
    } else {
      if (k < a.nr) sr[k * TPB + threadIdx.x] = a.r[i];
      if (k < a.nx) sx[k * TPB + threadIdx.x] = a.x[i];
      if (k < a.nc) scd[k * TPB + threadIdx.x] = a.C ? a.C[i] : 1.0;
    }
  }
  // p is read across CTAs; a cluster's sums need all of its CTAs started.
  if (PERM || CLUSTER) ok = sync_over<CLUSTER, TPB>(a.red, round);
  // C of step k: shared, global, or 1 (1 * r is r, exactly).
  auto c_at = [&](int k, int i) {
    return k < a.nc ? scd[k * TPB + threadIdx.x] : a.C ? __ldca(a.C + i) : 1.0;
  };
  // f(tag, k, i) over this thread's rows, two steps per call while there are
  // two, so that the loads of both are issued before the first store.
  auto rows2 = [&](auto f) {
    int k = 0, i = i0;
    for (; k + 1 < steps && i + stride < N; k += 2, i += 2 * stride) f(IntTag<2>{}, k, i);
    if (k < steps && i < N) f(IntTag<1>{}, k, i);
  };

  // fused: the preconditioned residual and the last direction that phase A
  // reads (the first time both are the setup's p, with a = b = 0), and the
  // direction it writes.
  const double *zc = a.p, *po = a.p;
  double *pn = a.p2;
  while (ok) {
    // A
    double s1[1] = {0.0};
    if constexpr (FUSED) {
      for (int k = 0, i = i0; k < steps && i < N; k++, i += stride) {
        const double poi = __ldca(po + i), pi = madd(__ldca(zc + i), beta, poi);
        const double qi =
            A.row(i, [&](int j) { return madd(__ldca(zc + j), beta, __ldca(po + j)); });
        double *xp = vec_at<TPB>(sx, a.nx, a.x, k, i);
        *xp = madd(*xp, alpha, poi);
        pn[i] = pi;
        *vec_at<TPB>(sq, a.nq, a.q, k, i) = qi;
        s1[0] = fma(pi, qi, s1[0]);
      }
    } else {
      const double *p = a.p;
      auto x_at = [&](int j) { return __ldca(p + j); };
      auto put = [&](int k, int i, double pi, double qi) {
        *vec_at<TPB>(sq, a.nq, a.q, k, i) = qi;
        s1[0] = fma(pi, qi, s1[0]);
      };
      if constexpr (PERM) {
        slice_rows<TPB, kSliceInFlight>(A.S, steps, x_at, put);
      } else {
        for (int k = 0, i = i0; k < steps && i < N; k++, i += stride) {
          A.prefetch(i, stride);
          const double pi = __ldca(p + i);
          put(k, i, pi, A.row(i, x_at));
        }
      }
    }
    ok = sum_over<CLUSTER, TPB, 1>(a.red, round, s1, sc, [&](const double (&s)[1], double *o) {
      o[0] = rho / s[0];
      o[1] = s[0];
    });
    if (!ok) break;
    alpha = sc[0];
    // B
    double s2[2] = {0.0, 0.0};
    rows2([&](auto tag, int k, int i) {
      constexpr int UB = decltype(tag)::value;
      double rv[UB], qv[UB], cv[UB];
      double *rp[UB];
#pragma unroll
      for (int u = 0; u < UB; u++) {
        const int iu = i + u * stride;
        rp[u] = vec_at<TPB>(sr, a.nr, a.r, k + u, iu);
        rv[u] = *rp[u];
        qv[u] = *vec_at<TPB>(sq, a.nq, a.q, k + u, iu);
        cv[u] = c_at(k + u, iu);
      }
#pragma unroll
      for (int u = 0; u < UB; u++) {
        const double ri = madd(rv[u], -alpha, qv[u]);
        const double zi = __dmul_rn(cv[u], ri);
        *rp[u] = ri;
        if (FUSED) a.z[i + u * stride] = zi;
        s2[0] = fma(ri, ri, s2[0]);
        s2[1] = fma(ri, zi, s2[1]);
      }
    });
    it++;
    ok = sum_over<CLUSTER, TPB, 2>(a.red, round, s2, sc + 2, [&](const double (&s)[2], double *o) {
      o[0] = sqrt(s[0]) / nrm0;
      o[1] = s[1] / rho;
      o[2] = s[1];
      o[3] = s[0];
    });
    if (!ok) break;
    if (FUSED) {
      double *t = pn;
      pn = po == zc ? a.p : const_cast<double *>(po);
      po = t;
      zc = a.z;
    }
    bool stop = sc[2] <= tol;
    if (stop) {
      conv = 1;
    } else {
      rho_old = rho;
      beta = sc[3];
      rho = sc[4];
      stop = it >= maxit;
    }
    if constexpr (FUSED) {
      if (stop) break;
    } else {
      // E: also in the iteration that stops, without the new direction.
      rows2([&](auto tag, int k, int i) {
        constexpr int UB = decltype(tag)::value;
        double rv[UB], xv[UB], pv[UB], cv[UB];
        double *xp[UB];
#pragma unroll
        for (int u = 0; u < UB; u++) {
          const int iu = i + u * stride;
          rv[u] = *vec_at<TPB>(sr, a.nr, a.r, k + u, iu);
          xp[u] = vec_at<TPB>(sx, a.nx, a.x, k + u, iu);
          xv[u] = *xp[u];
          pv[u] = __ldca(a.p + iu);
          cv[u] = c_at(k + u, iu);
        }
#pragma unroll
        for (int u = 0; u < UB; u++) {
          *xp[u] = madd(xv[u], alpha, pv[u]);
          if (!stop) a.p[i + u * stride] = madd(__dmul_rn(cv[u], rv[u]), beta, pv[u]);
        }
      });
      if (stop || !(ok = sync_over<CLUSTER, TPB>(a.red, round))) break;
    }
  }

  if (CLUSTER) cluster_sync();
  // Back to the global vectors; fused: the last x update and p.
  for (int k = 0, i = i0; k < steps && i < N; k++, i += stride) {
    double *xp = vec_at<TPB>(sx, a.nx, a.x, k, i);
    if (FUSED && ok) {
      const double pi = __ldca(po + i);
      *xp = madd(*xp, alpha, pi);
      if (po != a.p) a.p[i] = pi;
    }
    if constexpr (PERM) {
      const int j = A.from(i);
      a.xo[j] = *xp;
      a.ro[j] = *vec_at<TPB>(sr, a.nr, a.r, k, i);
      a.qo[j] = *vec_at<TPB>(sq, a.nq, a.q, k, i);
      a.po[j] = a.p[i];
    } else {
      if (k < a.nx) a.x[i] = *xp;
      if (k < a.nr) a.r[i] = sr[k * TPB + threadIdx.x];
      if (k < a.nq) a.q[i] = sq[k * TPB + threadIdx.x];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->r2 = sc[5];
    st->pq = sc[1];
    st->rho = rho;
    st->rho_old = rho_old;
    st->alpha = alpha;
    st->beta = beta;
    st->residual = sc[2];
    st->iteration = it;
    st->converged = conv;
    st->stop = 1;
    st->finished = 1;
  }
  if (!ok && threadIdx.x == 0) atomicOr(&st->error, kErrGridSync);
}

}  // namespace cgx

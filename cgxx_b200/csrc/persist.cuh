// Persistent inner solves of the mixed paths.
//
// Each inner FP32 PCG of a refinement step is one cooperative launch instead
// of a graph of four or five kernels per iteration: the CTAs (one per SM, all
// resident) run the phases of an iteration over the rows and meet at
// grid-wide barriers that carry the phase's dot products (gridred.cuh), so
// all CTAs hold the same alpha, beta and residual and take the same stop
// decision.
//
// Split form, one product or one update per phase, rows dealt to the CTAs in
// tiles of TPB, tile by tile:
//   learned: A  q = A p                         | <p,q> -> a
//            B  r -= a q                        | <r,r> -> test
//            C  y = G^T r                       |
//            D  z = G y + eps C r               | <r,z> -> b
//            E  d += a p, p = z + b p           |
//   Jacobi:  A  as above                        | <p,q> -> a
//            B  r -= a q                        | <r,r>, <r,Cr> -> test, b
//            E  d += a p, p = C r + b p         |
// Vectors that no other CTA reads (learned z, d, q and a second copy of r;
// Jacobi r, d, C, q) stay in shared memory for the whole launch, as many tiles
// of them as fit in kInnerResident; their order is by the traffic a byte saves.
//
// Fused form, a contiguous range of rows per CTA:
//   A  p = z + b p_old, d += a_old p_old, q = A p       | <p,q> -> a
//   B  learned: r = r_old - a q, y = G^T r              | (the CTAs below)
//      Jacobi:  r -= a q, z = C r                       | <r,r>, <r,z> -> test, b
//   C  learned: z = G y + eps C r                       | <r,r>, <r,z> -> test, b
// p and r are formed again at every neighbour the products read (in turn with
// the last ones' buffers), which saves barriers. Phase C reads y only of its
// own rows and of rows up to the largest offset before them, so between B and
// C a CTA waits for the few CTAs below it, not for the grid.
//
// The arithmetic is the graph iteration's (k_band, k_gband, k_inner_update,
// k_inner_direction): the same products added in the same order. The band
// values, the factor and C do not change during a launch and take the
// read-only path (__ldg). The vectors are written inside the launch and are
// read with weak loads (ldv): every read of another CTA's value comes after a
// barrier whose GPU-scope acquire makes that value visible to the weak loads
// that follow it, so L1 holds no line from before the barrier that is still
// read. (Reading them through L2 only, __ldcg, measured 1-2 % slower.)
//
// What bounds it: at 96^3 and below the barriers (2.1-2.3 us each with the
// CTAs' skew) and the bytes through L1 (190 read and 110 filled per row of a
// fused learned iteration, 84 % of the L1 data banks' cycles in its phases); at
// 160^3 DRAM and L2. One CTA per SM (128 registers at 512 threads, 64 at 1024:
// two rows in flight per thread), one warp that does each barrier's sums, and
// resident vectors took the iteration (us) from 12.4 to 11.3 (96^3 Jacobi), 21.7
// to 17.7 (128^3), 45.0 to 38.1 (160^3), and learned 18.2 to 16.4 and 41.0 to 32.5;
// 24^3: 7.5 to 4.8 and 9.3 to 6.6. At 160^3 learned they are level (69.1 before, 68.3
// to 70 now), although DRAM carries 227 MB an iteration instead of 268.
//
// Every wait of a cooperative launch is bounded: a CTA that gives up sets
// kErrGridSync in CgState::error and leaves the loop, so the launch always ends
// and the host reports CGX_ERROR_DEVICE. A cluster launch waits at the hardware's
// cluster barrier, which has no limit: all of its CTAs run together and take the
// same decisions from the same sums, so each of them reaches every barrier.
#pragma once

#include "band.cuh"
#include "gridred.cuh"
#include "kernels.cuh"
#include "offsets.cuh"
#include "sell.cuh"
#include "slices.cuh"

namespace cgx {

// Shared memory given to resident vectors; the rest stays L1 for the gathers.
constexpr int kInnerResident = 192 << 10;

__device__ __forceinline__ float ldv(const float *p) { return __ldca(p); }

// Diagnostics of the bounded waits: waits that nothing can complete, with a
// short limit, so that the give-up path runs and sets its error bit.
//  - a grid barrier that one of the launch's two CTAs never reaches;
//  - an mbarrier (one expected arrival) that nobody arrives on.
__global__ void __launch_bounds__(128) k_wait_timeout(RedMem *red, int which, unsigned polls,
                                                      CgState *st) {
  if (which == 0) {
    unsigned round = 0;
    if (blockIdx.x == 0 && !grid_barrier<128>(red, round, polls) && threadIdx.x == 0)
      atomicOr(&st->error, kErrGridSync);
    return;
  }
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  if (!mbar_wait_bounded(&bar, 0u, polls) && threadIdx.x == 0)
    atomicOr(&st->error, kErrBarrierTimeout);
}

struct InnerArgs {
  float *p, *p2;   // the direction; fused: in turn
  float *r, *r2;   // the residual; fused learned: in turn
  float *z, *d, *q;
  float *y;        // learned: G^T r
  const float *C;  // FP32 Jacobi vector
  float eps;       // learned: eps of eps C r
  RedMem *red;     // zeroed (kRedZeroBytes) before the launch
  int steps;       // tiles (split) or passes (fused) per CTA
  int rows;        // fused: rows per CTA
  int below;       // fused learned: CTAs below whose y phase C reads
  int nz, nr, nd, nq, nc;  // tiles or passes held in shared memory
  // Sorted slices: r, p, C and d in the matrix's own row order; the vectors above
  // are in slot order.
  const float *ro, *po, *Co;
  float *dout;
};

// Scalars of the loop, shared by a CTA's threads: sc[0] alpha, sc[1] residual,
// sc[2] beta, sc[3] rho.
struct InnerLoop {
  double rho, nrm0, tol;
  int it = 0, total, maxit;
  __device__ explicit InnerLoop(const CgState *st)
      : rho(st->in_rho), nrm0(st->in_nrm0), tol(st->in_tol), total(st->total_inner),
        maxit(st->max_iter) {}
  // The iteration's stop test (inner_broke_down and the residual test of the
  // graph's k_inner_update).
  __device__ bool stop(double res, double alpha) {
    it++;
    total++;
    return !(res > tol) || !(fabs(alpha) <= 1.7976931348623157e308) || alpha == 0.0 ||
           total >= maxit;
  }
  __device__ void publish(CgState *st, const double *sc, double alpha, double beta,
                          bool ok) const {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->in_alpha = alpha;
      st->in_beta = beta;
      st->in_rho = rho;
      st->in_res = sc[1];
      st->in_iter = it;
      st->total_inner = total;
      st->in_stop = 1;
      st->in_finished = 1;
    }
    if (!ok && threadIdx.x == 0) atomicOr(&st->error, kErrGridSync);
  }
};

// --- the products' rows ------------------------------------------------------

// A vector that is stored, and s a + b formed where it is read.
struct Stored {
  const float *v;
  __device__ float operator()(int i) const { return ldv(v + i); }
};
struct Combined {
  float s;
  const float *a, *b;
  __device__ float operator()(int i) const { return fmaf(s, ldv(a + i), ldv(b + i)); }
};

// Row i of A times x; xi = element i. (Values by offset instead of by row, and
// rows without clamps and masks in the interior, measured no gain: with the
// vectors in L2 the products are bound by the bytes that go through L1, 190
// read and 110 filled per row of a fused learned iteration, not by the
// instructions.)
template <typename X>
__device__ __forceinline__ float band_row(const BandView<4> &B, int i, float xi, const X &x) {
  const unsigned nmax = (unsigned)(B.N - 1);
  const float4 u = __ldg(reinterpret_cast<const float4 *>(B.U) + i);
  float xu[4], lv[4], xl[4];
  xu[0] = xi;
#pragma unroll
  for (int k = 1; k < 4; k++) {
    xu[k] = x((int)min((unsigned)i + (unsigned)B.d[k], nmax));
    const int j = i - B.d[k], jc = max(j, 0);
    lv[k] = __ldg(&B.U[(size_t)jc * 4 + k]);
    xl[k] = x(jc);
    lv[k] = j < 0 ? 0.f : lv[k];
  }
  float sum = fmaf(u.x, xu[0], 0.f);
  sum = fmaf(u.y, xu[1], sum);
  sum = fmaf(u.z, xu[2], sum);
  sum = fmaf(u.w, xu[3], sum);
#pragma unroll
  for (int k = 1; k < 4; k++) sum = fmaf(lv[k], xl[k], sum);
  return sum;
}

// Row i of G^T times x; xi = element i.
template <typename X>
__device__ __forceinline__ float gband_t_row(const GBandView &B, int i, float xi, const X &x) {
  const unsigned short *gv = reinterpret_cast<const unsigned short *>(B.val);
  float v[4], xv[4];
  v[0] = bf16_bits_to_float(__ldg(&gv[(size_t)i * 4]));
  xv[0] = xi;
#pragma unroll
  for (int k = 1; k < 4; k++) {
    const unsigned j = (unsigned)i + (unsigned)B.d[k];
    const int jc = (int)min(j, (unsigned)(B.N - 1));
    v[k] = bf16_bits_to_float(__ldg(&gv[(size_t)jc * 4 + k]));
    xv[k] = x(jc);
    v[k] = j < (unsigned)B.N ? v[k] : 0.f;
  }
  float sum = 0.f;
#pragma unroll
  for (int k = 0; k < 4; k++) sum = fmaf(v[k], xv[k], sum);
  return sum;
}

// Row i of G times y.
__device__ __forceinline__ float gband_row(const GBandView &B, int i, const float *y) {
  const uint2 raw = __ldg(reinterpret_cast<const uint2 *>(B.val) + i);
  const float v[4] = {__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u),
                      __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u)};
  float xv[4], sum = 0.f;
#pragma unroll
  for (int k = 0; k < 4; k++) xv[k] = ldv(y + max(i - B.d[k], 0));
#pragma unroll
  for (int k = 0; k < 4; k++) sum = fmaf(v[k], xv[k], sum);
  return sum;
}

// L2 prefetch of read-only row values two tiles ahead, one lane per 128-byte
// line: more of the band stream in flight than the warps' registers hold.
template <int BYTES_PER_ROW>
__device__ __forceinline__ void prefetch_row(const void *base, int i, int stride, int N) {
  constexpr int kRowsPerLine = 128 / BYTES_PER_ROW;
  const long long j = (long long)i + 2ll * stride;
  if ((threadIdx.x & (kRowsPerLine - 1)) == 0 && j < N)
    asm volatile("prefetch.global.L2 [%0];"
                 :
                 : "l"((const char *)base + j * BYTES_PER_ROW));
}

// --- split form --------------------------------------------------------------

// Streaming phases: four consecutive rows per thread. f4(tile, o, i) handles
// rows i .. i + 3 of a tile at offset o in it; f1 the last N mod 4 rows.
template <int TPB, typename F4, typename F1>
__device__ __forceinline__ void tile_quads(int N, int steps, F4 f4, F1 f1) {
  static_assert(TPB % 128 == 0, "tile_quads");
  constexpr int Q = TPB / 4;  // quads per tile
  const int o = 4 * ((int)threadIdx.x % Q);
  for (int k = (int)threadIdx.x / Q; k < steps; k += 4) {
    const long long i = ((long long)k * gridDim.x + blockIdx.x) * TPB + o;
    if (i + 4 <= N)
      f4(k, o, (int)i);
    else
      for (int j = 0; j < 4 && i + j < N; j++) f1(k, o + j, (int)i + j);
  }
}

// Tile k of a vector: the first n tiles in shared memory, the rest global.
template <int TPB>
__device__ __forceinline__ float *tile_at(float *sm, int n, float *g, int k, int o, int i) {
  return k < n ? sm + (k * TPB + o) : g + i;
}
__device__ __forceinline__ float4 quad(const float *p) {
  return *reinterpret_cast<const float4 *>(p);
}
__device__ __forceinline__ void quad_to(float *p, float4 v) {
  *reinterpret_cast<float4 *>(p) = v;
}
__device__ __forceinline__ float4 fma4(float a, float4 x, float4 y) {
  return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}
__device__ __forceinline__ float4 mul4(float4 x, float4 y) {
  return make_float4(x.x * y.x, x.y * y.y, x.z * y.z, x.w * y.w);
}
__device__ __forceinline__ double dot4(float4 x, float4 y, double s) {
  s = fma((double)x.x, (double)y.x, s);
  s = fma((double)x.y, (double)y.y, s);
  s = fma((double)x.z, (double)y.z, s);
  return fma((double)x.w, (double)y.w, s);
}

// The matrix-dependent phases of the split form. Band: A and G on the band.
template <bool LEARNED, bool PF, int TPB>
struct BandPhases {
  static constexpr bool kLearned = LEARNED;
  // q (and z) of a tile may be kept in shared memory: the thread that writes
  // row i of a product is the tile's, so the tile stays in its CTA.
  static constexpr bool kTiled = true;
  static constexpr bool kPerm = false;
  BandView<4> A;
  GBandView G;
  __device__ int N() const { return A.N; }
  // f(tag, k, i, stride): row i of tile k and, for tag 2, row i + stride of
  // the next tile, whose loads are issued before the first store.
  template <typename F>
  __device__ void rows2(int steps, F f) const {
    const int stride = gridDim.x * TPB;
    int k = 0, i = blockIdx.x * TPB + threadIdx.x;
    for (; k + 1 < steps && i + stride < A.N; k += 2, i += 2 * stride)
      f(IntTag<2>{}, k, i, stride);
    if (k < steps && i < A.N) f(IntTag<1>{}, k, i, stride);
  }
  // q = A p; returns the partial of <p,q>.
  __device__ double q_rows(const InnerArgs &a, float *sq) const {
    double s = 0.0;
    const float *p = a.p;
    rows2(a.steps, [&](auto tag, int k, int i, int stride) {
      constexpr int UB = decltype(tag)::value;
      float pv[UB], qv[UB];
#pragma unroll
      for (int u = 0; u < UB; u++) {
        const int iu = i + u * stride;
        if (PF) prefetch_row<16>(A.U, iu, stride, A.N);
        pv[u] = ldv(p + iu);
        qv[u] = band_row(A, iu, pv[u], Stored{p});
      }
#pragma unroll
      for (int u = 0; u < UB; u++) {
        *tile_at<TPB>(sq, a.nq, a.q, k + u, threadIdx.x, i + u * stride) = qv[u];
        s = fma((double)pv[u], (double)qv[u], s);
      }
    });
    return s;
  }
  __device__ void y_rows(const InnerArgs &a) const {
    const float *r = a.r;
    rows2(a.steps, [&](auto tag, int, int i, int stride) {
      constexpr int UB = decltype(tag)::value;
      float yv[UB];
#pragma unroll
      for (int u = 0; u < UB; u++) {
        const int iu = i + u * stride;
        if (PF) prefetch_row<8>(G.val, iu, stride, A.N);
        yv[u] = gband_t_row(G, iu, ldv(r + iu), Stored{r});
      }
#pragma unroll
      for (int u = 0; u < UB; u++) a.y[i + u * stride] = yv[u];
    });
  }
  // z = G y + eps C r; returns the partial of <r,z>.
  __device__ double z_rows(const InnerArgs &a, float *sz, float *sr) const {
    double s = 0.0;
    rows2(a.steps, [&](auto tag, int k, int i, int stride) {
      constexpr int UB = decltype(tag)::value;
      float rv[UB], zv[UB];
#pragma unroll
      for (int u = 0; u < UB; u++) {
        const int iu = i + u * stride;
        if (PF) prefetch_row<8>(G.val, iu, stride, A.N);
        rv[u] = *tile_at<TPB>(sr, a.nr, a.r, k + u, threadIdx.x, iu);
        zv[u] = fmaf(a.eps * __ldg(a.C + iu), rv[u],
                     gband_row(G, iu, a.y));
      }
#pragma unroll
      for (int u = 0; u < UB; u++) {
        *tile_at<TPB>(sz, a.nz, a.z, k + u, threadIdx.x, i + u * stride) = zv[u];
        s = fma((double)rv[u], (double)zv[u], s);
      }
    });
    return s;
  }
};

// Row i of a symmetric A stored by offset (lower values from the mirror rows)
// times x, in ascending column order; x is finite, so an entry that a row does
// not have (value 0) adds nothing. The loads of a group of slots are issued
// before its sums.
template <int K, typename X>
__device__ __forceinline__ float offset_row(const Band64View<K, true, float> &B, int i, const X &x) {
  const float *__restrict__ U = B.U;
  const unsigned nmax = (unsigned)(B.N - 1);
  constexpr int kSlots = 2 * K - 1, G = 7;
  float sum = 0.f;
#pragma unroll
  for (int s0 = 0; s0 < kSlots; s0 += G) {
    float v[G], xv[G];
#pragma unroll
    for (int g = 0; g < G; g++) {
      const int s = s0 + g;
      if (s >= kSlots) continue;
      if (s < K - 1) {
        const int k = K - 1 - s, j = i - B.d[k], jc = max(j, 0);
        v[g] = __ldg(U + k * B.ld + jc);
        xv[g] = x(jc);
        v[g] = j < 0 ? 0.f : v[g];
      } else {
        const int k = s - (K - 1);
        v[g] = __ldg(U + k * B.ld + i);
        xv[g] = x((int)min((unsigned)(i + B.d[k]), nmax));
      }
    }
#pragma unroll
    for (int g = 0; g < G; g++)
      if (s0 + g < kSlots) sum = fmaf(v[g], xv[g], sum);
  }
  return sum;
}

// A by offset (Jacobi only): half the value bytes of the uniform slices. Bound by
// L2's throughput, as the mirror values of the plane below come from there: at
// 128^3 about 108 bytes a row and product, 226 MB in 36 us. us per iteration of
// 27-point grids, uniform slices -> by offset: 24^3 10.9 -> 7.3, 48^3 14.2 -> 8.7,
// 64^3 15.8 -> 11.4, 96^3 28.6 -> 20.1, 128^3 55.2 -> 44.0. (Groups of 7, 9 or 14
// slots, L2 prefetch of the next step's values, 128 or 160 KB of resident vectors:
// within 1 us.)
template <int K, int TPB>
struct OffsetPhases {
  static constexpr bool kLearned = false;
  static constexpr bool kTiled = true;
  static constexpr bool kPerm = false;
  Band64View<K, true, float> A;
  __device__ int N() const { return A.N; }
  __device__ double q_rows(const InnerArgs &a, float *sq) const {
    double s = 0.0;
    const float *p = a.p;
    const int stride = gridDim.x * TPB;
    for (int k = 0, i = blockIdx.x * TPB + threadIdx.x; k < a.steps && i < A.N; k++, i += stride) {
      const float pv = ldv(p + i), qv = offset_row(A, i, Stored{p});
      *tile_at<TPB>(sq, a.nq, a.q, k, threadIdx.x, i) = qv;
      s = fma((double)pv, (double)qv, s);
    }
    return s;
  }
  __device__ void y_rows(const InnerArgs &) const {}
  __device__ double z_rows(const InnerArgs &, float *, float *) const { return 0.0; }
};

// SELL-U: A, G and G^T in uniform slices (sell.cuh). Its products deal slices,
// not tiles, to the warps, so q, z and the r they read are global.
// AOFF: A by offset, whose product deals rows in tiles.
template <bool LEARNED, bool AOFF, int TPB>
struct SellPhases {
  static constexpr bool kLearned = LEARNED;
  static constexpr bool kTiled = false;
  static constexpr bool kPerm = false;
  static constexpr int U = 8;
  SellUView<float> A;
  SellUView<__nv_bfloat16> G, GT;
  Band64View<kBand64MaxHalf, true, float> AO;
  struct OpQ {  // q = A p, <p,q>
    using Acc = Acc1;
    struct Pre {
      float p;
    };
    const float *p;
    float *q;
    __device__ Pre prefetch(int i) const { return Pre{ldv(p + i)}; }
    __device__ void row(int i, float s, Acc &a, const Pre &pr) const {
      q[i] = s;
      a.a0 = fma((double)pr.p, (double)s, a.a0);
    }
  };
  struct OpZ {  // z = G y + eps C r, <r,z> (OpLearnedZ's arithmetic)
    using Acc = Acc1;
    struct Pre {
      float r, c;
    };
    const float *r, *C;
    float *z;
    float eps;
    __device__ Pre prefetch(int i) const { return Pre{ldv(r + i), __ldg(C + i)}; }
    __device__ void row(int i, float s, Acc &a, const Pre &pr) const {
      const float zi = fmaf(eps * pr.c, pr.r, s);
      z[i] = zi;
      a.a0 = fma((double)pr.r, (double)zi, a.a0);
    }
  };
  __device__ int N() const { return A.N; }
  __device__ double q_rows(const InnerArgs &a, float *) const {
    if constexpr (AOFF) return OffsetPhases<kBand64MaxHalf, TPB>{AO}.q_rows(a, nullptr);
    Acc1 acc;
    sellu_rows<float, U, true, TPB>(A, a.p, GatherWeak{}, OpQ{a.p, a.q}, acc);
    return acc.a0;
  }
  __device__ void y_rows(const InnerArgs &a) const {
    NoAcc none;
    sellu_rows<__nv_bfloat16, U, true, TPB>(GT, a.r, GatherWeak{}, OpInnerStore{a.y}, none);
  }
  __device__ double z_rows(const InnerArgs &a, float *, float *) const {
    Acc1 acc;
    sellu_rows<__nv_bfloat16, U, true, TPB>(G, a.y, GatherWeak{}, OpZ{a.r, a.C, a.z, a.eps},
                                            acc);
    return acc.a0;
  }
};

// Sorted slices (slices.cuh), for irregular matrices: a slot's rows of all the
// products belong to the same tile.
template <bool LEARNED, int TPB>
struct SlicePhases {
  static constexpr bool kLearned = LEARNED;
  static constexpr bool kTiled = true;
  static constexpr bool kPerm = true;
  SliceView<float> A;
  SliceView<__nv_bfloat16> G, GT;
  const int *perm;
  __device__ int N() const { return A.N; }
  __device__ double q_rows(const InnerArgs &a, float *sq) const {
    double s = 0.0;
    slice_rows<TPB, kSliceInFlight32>(
        A, a.steps, [&](int j) { return ldv(a.p + j); },
        [&](int k, int i, float pv, float qv) {
          *tile_at<TPB>(sq, a.nq, a.q, k, threadIdx.x, i) = qv;
          s = fma((double)pv, (double)qv, s);
        });
    return s;
  }
  __device__ void y_rows(const InnerArgs &a) const {
    slice_rows<TPB, kSliceInFlight32>(
        GT, a.steps, [&](int j) { return ldv(a.r + j); },
        [&](int, int i, float, float yv) { a.y[i] = yv; });
  }
  __device__ double z_rows(const InnerArgs &a, float *sz, float *sr) const {
    double s = 0.0;
    slice_rows<TPB, kSliceInFlight32>(
        G, a.steps, [&](int j) { return ldv(a.y + j); },
        [&](int k, int i, float, float gy) {
          const float rv = *tile_at<TPB>(sr, a.nr, a.r, k, threadIdx.x, i);
          const float zv = fmaf(a.eps * ldv(a.C + i), rv, gy);
          *tile_at<TPB>(sz, a.nz, a.z, k, threadIdx.x, i) = zv;
          s = fma((double)rv, (double)zv, s);
        });
    return s;
  }
};

template <typename Phases, bool CLUSTER, int TPB>
__global__ void __launch_bounds__(TPB, 1)
    k_inner_split(Phases P, InnerArgs a, CgState *st) {
  constexpr bool LEARNED = Phases::kLearned;
  extern __shared__ __align__(16) float smf[];
  __shared__ double sc[4];
  float *const sz = smf;
  float *const sr = sz + (size_t)a.nz * TPB;
  float *const sd = sr + (size_t)a.nr * TPB;
  float *const sq = sd + (size_t)a.nd * TPB;
  float *const scd = sq + (size_t)a.nq * TPB;
  const int N = P.N(), steps = a.steps;
  InnerLoop loop(st);
  double alpha = 0.0, beta = 0.0;
  unsigned round = 0;
  bool ok = true;

  // Resident vectors that hold values at the start.
  auto bring = [&](float *sm, int n, const float *g) {
    for (int k = 0; k < n; k++) {
      const long long i = ((long long)k * gridDim.x + blockIdx.x) * TPB + threadIdx.x;
      if (i < N) sm[k * TPB + threadIdx.x] = g[i];
    }
  };
  if constexpr (Phases::kPerm) {
    for (int k = 0; k < steps; k++) {
      const long long l = ((long long)k * gridDim.x + blockIdx.x) * TPB + threadIdx.x;
      if (l >= N) break;
      const int i = (int)l, j = __ldg(P.perm + i), t = threadIdx.x;
      *tile_at<TPB>(sr, a.nr, a.r, k, t, i) = a.ro[j];
      *tile_at<TPB>(sd, a.nd, a.d, k, t, i) = 0.f;
      *tile_at<TPB>(scd, a.nc, const_cast<float *>(a.C), k, t, i) = a.Co[j];
      a.p[i] = a.po[j];
    }
    ok = sync_over<CLUSTER, TPB>(a.red, round);  // p is read across CTAs
  } else {
    bring(sr, a.nr, a.r);
    bring(sd, a.nd, a.d);
    bring(scd, a.nc, a.C);
    if (CLUSTER)
      cluster_sync();  // cluster_sum needs all of its CTAs started
    else
      __syncthreads();
  }
  // C is written in this launch only with kPerm (then not the read-only path).
  auto cval = [&](int k, int o, int i) {
    return !Phases::kPerm ? __ldg(a.C + i) : k < a.nc ? scd[k * TPB + o] : ldv(a.C + i);
  };
  auto c4 = [&](int i) {
    const float4 *c = reinterpret_cast<const float4 *>(a.C + i);
    return Phases::kPerm ? *c : __ldg(c);
  };

  while (ok) {
    // A
    {
      const double s[1] = {P.q_rows(a, sq)};
      ok = sum_over<CLUSTER, TPB, 1>(a.red, round, s, sc,
                            [&](const double (&t)[1], double *o) { o[0] = loop.rho / t[0]; });
      if (!ok) break;
      alpha = sc[0];
    }
    // B (the learned products read r of other rows: it is always stored to the
    // global vector too)
    {
      const float na = (float)(-alpha);
      double s[2] = {0.0, 0.0};
      tile_quads<TPB>(
          N, steps,
          [&](int k, int o, int i) {
            float *rp = tile_at<TPB>(sr, a.nr, a.r, k, o, i);
            const float4 r0 = quad(rp), qv = quad(tile_at<TPB>(sq, a.nq, a.q, k, o, i));
            const float4 cv = LEARNED ? r0
                              : k < a.nc ? quad(scd + (k * TPB + o))
                                         : c4(i);
            const float4 rv = fma4(na, qv, r0);
            quad_to(rp, rv);
            if (LEARNED && k < a.nr) quad_to(a.r + i, rv);
            s[0] = dot4(rv, rv, s[0]);
            if (!LEARNED) s[1] = dot4(rv, mul4(cv, rv), s[1]);
          },
          [&](int k, int o, int i) {
            float *rp = tile_at<TPB>(sr, a.nr, a.r, k, o, i);
            const float rv = fmaf(na, *tile_at<TPB>(sq, a.nq, a.q, k, o, i), *rp);
            *rp = rv;
            if (LEARNED && k < a.nr) a.r[i] = rv;
            s[0] = fma((double)rv, (double)rv, s[0]);
            if (!LEARNED) s[1] = fma((double)rv, (double)(cval(k, o, i) * rv), s[1]);
          });
      if (LEARNED) {
        const double s1[1] = {s[0]};
        ok = sum_over<CLUSTER, TPB, 1>(a.red, round, s1, sc + 1, [&](const double (&t)[1], double *o) {
          o[0] = sqrt(t[0]) / loop.nrm0;
        });
      } else {
        ok = sum_over<CLUSTER, TPB, 2>(a.red, round, s, sc + 1, [&](const double (&t)[2], double *o) {
          o[0] = sqrt(t[0]) / loop.nrm0;
          o[1] = t[1] / loop.rho;
          o[2] = t[1];
        });
      }
      if (!ok) break;
    }
    const bool stop = loop.stop(sc[1], alpha);
    if (LEARNED && !stop) {
      P.y_rows(a);
      if (!(ok = sync_over<CLUSTER, TPB>(a.red, round))) break;
      const double s[1] = {P.z_rows(a, sz, sr)};
      ok = sum_over<CLUSTER, TPB, 1>(a.red, round, s, sc + 2, [&](const double (&t)[1], double *o) {
        o[0] = t[0] / loop.rho;
        o[1] = t[0];
      });
      if (!ok) break;
    }
    if (!stop) {
      beta = sc[2];
      loop.rho = sc[3];
    }
    // E: also in the iteration that stops, without the new direction.
    {
      const float al = (float)alpha, be = (float)beta;
      tile_quads<TPB>(
          N, steps,
          [&](int k, int o, int i) {
            float *dp = tile_at<TPB>(sd, a.nd, a.d, k, o, i);
            const float4 pv = quad(a.p + i), dv = quad(dp);
            float4 zv;
            if (LEARNED) {
              zv = quad(tile_at<TPB>(sz, a.nz, a.z, k, o, i));
            } else {
              const float4 rv = quad(tile_at<TPB>(sr, a.nr, a.r, k, o, i));
              const float4 cv = k < a.nc ? quad(scd + (k * TPB + o)) : c4(i);
              zv = mul4(cv, rv);
            }
            quad_to(dp, fma4(al, pv, dv));
            if (!stop) quad_to(a.p + i, fma4(be, pv, zv));
          },
          [&](int k, int o, int i) {
            float *dp = tile_at<TPB>(sd, a.nd, a.d, k, o, i);
            const float pi = ldv(a.p + i);
            const float zi = LEARNED ? *tile_at<TPB>(sz, a.nz, a.z, k, o, i)
                                     : cval(k, o, i) * *tile_at<TPB>(sr, a.nr, a.r, k, o, i);
            *dp = fmaf(al, pi, *dp);
            if (!stop) a.p[i] = fmaf(be, pi, zi);
          });
    }
    if (stop || !(ok = sync_over<CLUSTER, TPB>(a.red, round))) break;
  }
  if (CLUSTER) cluster_sync();
  // d is what the refinement step needs.
  __syncthreads();
  if constexpr (Phases::kPerm) {
    for (int k = 0; k < steps; k++) {
      const long long l = ((long long)k * gridDim.x + blockIdx.x) * TPB + threadIdx.x;
      if (l >= N) break;
      a.dout[__ldg(P.perm + (int)l)] = *tile_at<TPB>(sd, a.nd, a.d, k, threadIdx.x, (int)l);
    }
  } else {
    for (int k = 0; k < a.nd; k++) {
      const long long i = ((long long)k * gridDim.x + blockIdx.x) * TPB + threadIdx.x;
      if (i < N) a.d[i] = sd[k * TPB + threadIdx.x];
    }
  }
  loop.publish(st, sc, alpha, beta, ok);
}

// --- fused form --------------------------------------------------------------

template <bool LEARNED, bool CLUSTER, int TPB>
__global__ void __launch_bounds__(TPB, 1)
    k_inner_fused(BandView<4> A, GBandView G, InnerArgs a, CgState *st) {
  extern __shared__ __align__(16) float smf[];
  __shared__ double sc[4];
  float *const sd = smf;
  float *const sc32 = sd + (size_t)a.nd * TPB;
  float *const sr = sc32 + (size_t)a.nc * TPB;
  float *const sq = sr + (size_t)a.nr * TPB;
  const int N = A.N, lo = blockIdx.x * a.rows, hi = min(N, lo + a.rows);
  InnerLoop loop(st);
  double alpha = 0.0, beta = 0.0;
  unsigned round = 0;
  bool ok = true;
  for (int k = 0, i = lo + threadIdx.x; i < hi; k++, i += TPB) {
    if (k < a.nd) sd[k * TPB + threadIdx.x] = a.d[i];
    if (k < a.nc) sc32[k * TPB + threadIdx.x] = a.C[i];
    if (k < a.nr) sr[k * TPB + threadIdx.x] = a.r[i];
  }
  auto at = [&](float *sm, int n, float *g, int k, int i) {
    return k < n ? sm + (k * TPB + (int)threadIdx.x) : g + i;
  };
  auto c_at = [&](int k, int i) {
    return k < a.nc ? sc32[k * TPB + threadIdx.x] : __ldg(a.C + i);
  };
  // f(tag, k, i): UB rows i, i + TPB, ... of passes k, k + 1, ..., whose loads
  // are issued before the first store.
  auto rows2 = [&](auto f) {
    int k = 0, i = lo + (int)threadIdx.x;
    for (; i + TPB < hi; k += 2, i += 2 * TPB) f(IntTag<2>{}, k, i);
    if (i < hi) f(IntTag<1>{}, k, i);
  };
  if (CLUSTER) cluster_sync();  // cluster_sum needs all of its CTAs started
  // The start's p = z: the first iteration forms p = z and leaves d at 0.
  const float *po = a.p, *ro = a.r;
  float *pn = a.p2, *rn = a.r2;
  const float *z = a.z;
  for (;;) {
    // A
    {
      const float al = (float)alpha, be = (float)beta;
      double s[1] = {0.0};
      const Combined pc{be, po, z};
      rows2([&](auto tag, int k, int i) {
        constexpr int UB = decltype(tag)::value;
        float pv[UB], qv[UB], ov[UB], dv[UB];
        float *dp[UB];
#pragma unroll
        for (int u = 0; u < UB; u++) {
          const int iu = i + u * TPB;
          ov[u] = ldv(po + iu);
          pv[u] = fmaf(be, ov[u], ldv(z + iu));
          qv[u] = band_row(A, iu, pv[u], pc);
          dp[u] = at(sd, a.nd, a.d, k + u, iu);
          dv[u] = *dp[u];
        }
#pragma unroll
        for (int u = 0; u < UB; u++) {
          const int iu = i + u * TPB;
          *dp[u] = fmaf(al, ov[u], dv[u]);
          pn[iu] = pv[u];
          *at(sq, a.nq, a.q, k + u, iu) = qv[u];
          s[0] = fma((double)pv[u], (double)qv[u], s[0]);
        }
      });
      ok = sum_over<CLUSTER, TPB, 1>(a.red, round, s, sc,
                            [&](const double (&t)[1], double *o) { o[0] = loop.rho / t[0]; });
      if (!ok) break;
      alpha = sc[0];
    }
    const float na = (float)(-alpha);
    double s[2] = {0.0, 0.0};
    if constexpr (LEARNED) {
      // B
      const Combined rc{na, a.q, ro};
      rows2([&](auto tag, int, int i) {
        constexpr int UB = decltype(tag)::value;
        float rv[UB], yv[UB];
#pragma unroll
        for (int u = 0; u < UB; u++) {
          const int iu = i + u * TPB;
          rv[u] = rc(iu);
          yv[u] = gband_t_row(G, iu, rv[u], rc);
        }
#pragma unroll
        for (int u = 0; u < UB; u++) {
          rn[i + u * TPB] = rv[u];
          a.y[i + u * TPB] = yv[u];
          s[0] = fma((double)rv[u], (double)rv[u], s[0]);
        }
      });
      if constexpr (CLUSTER)
        cluster_sync();
      else if (!(ok = wait_below<TPB>(a.red->flags, a.below, (unsigned long long)loop.it + 1)))
        break;
      // C
      rows2([&](auto tag, int k, int i) {
        constexpr int UB = decltype(tag)::value;
        float rv[UB], zv[UB];
#pragma unroll
        for (int u = 0; u < UB; u++) {
          const int iu = i + u * TPB;
          rv[u] = ldv(rn + iu);
          zv[u] = fmaf(a.eps * c_at(k + u, iu), rv[u],
                       gband_row(G, iu, a.y));
        }
#pragma unroll
        for (int u = 0; u < UB; u++) {
          a.z[i + u * TPB] = zv[u];
          s[1] = fma((double)rv[u], (double)zv[u], s[1]);
        }
      });
    } else {
      // B
      rows2([&](auto tag, int k, int i) {
        constexpr int UB = decltype(tag)::value;
        float rv[UB], zv[UB];
        float *rp[UB];
#pragma unroll
        for (int u = 0; u < UB; u++) {
          const int iu = i + u * TPB;
          rp[u] = at(sr, a.nr, a.r, k + u, iu);
          rv[u] = fmaf(na, *at(sq, a.nq, a.q, k + u, iu), *rp[u]);
          zv[u] = c_at(k + u, iu) * rv[u];
        }
#pragma unroll
        for (int u = 0; u < UB; u++) {
          *rp[u] = rv[u];
          a.z[i + u * TPB] = zv[u];
          s[0] = fma((double)rv[u], (double)rv[u], s[0]);
          s[1] = fma((double)rv[u], (double)zv[u], s[1]);
        }
      });
    }
    ok = sum_over<CLUSTER, TPB, 2>(a.red, round, s, sc + 1, [&](const double (&t)[2], double *o) {
      o[0] = sqrt(t[0]) / loop.nrm0;
      o[1] = t[1] / loop.rho;
      o[2] = t[1];
    });
    if (!ok) break;
    {
      float *t = const_cast<float *>(po);
      po = pn;
      pn = t;
      t = const_cast<float *>(ro);
      ro = rn;
      rn = t;
    }
    if (loop.stop(sc[1], alpha)) break;
    beta = sc[2];
    loop.rho = sc[3];
  }
  if (CLUSTER) cluster_sync();
  // d, with the update that phase A had still to make.
  const float al = (float)alpha;
  for (int k = 0, i = lo + threadIdx.x; i < hi; k++, i += TPB)
    a.d[i] = fmaf(al, ldv(po + i), *at(sd, a.nd, a.d, k, i));
  loop.publish(st, sc, alpha, beta, ok);
}

}  // namespace cgx

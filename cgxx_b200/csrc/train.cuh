// Training of the learned preconditioner's network: the Hutchinson loss
// ||(Ghat^T Ahat Ghat - I) V||^2 / (N S) over S probe columns (node-major:
// V[i * S + s]) and its gradient. No atomics, and every sum in one fixed
// order: the gradient is deterministic.
//
//   probes     V (Rademacher), smoothed columns                  k_smooth8
//   forward    network, Ghat (learned.cuh)
//   loss       T1 = Ghat V, T2 = Ahat T1, R = Ghat^T T2 - V      k_spmm8, k_loss_residual
//   backward   dT2 = Ghat rho, dT1 = Ahat dT2                    k_spmm8
//              dGhat, head outputs                               k_grad_rows, k_grad_cols
//              per layer: gradients of W_l, b_l, and of h_l      k_layer_back
//              embedding                                         k_embed_back
//              sums over the CTAs                                k_sum_partials
//
// The sparse kernels are bound by the 32-byte rows they gather: two lanes hold
// a row's halves, so that a warp's loads of one entry cover 16 rows, and a
// chunk's columns and values are loaded before its rows. A chunk's loads are
// unconditional (entries past the row's end re-read its last one, an L1 hit, and
// are left out of the sums): behind a condition each becomes a branch that waits
// for the load before it. At 96^3 (us, before -> after): k_spmm8 29 -> 24 on A and
// 24 -> 17 on G, k_loss_residual 35 -> 26, k_grad_rows 80 -> 63, k_embed_back 298
// -> 157.
#pragma once

#include <cfloat>

#include "learned.cuh"

namespace cgx {
namespace learned {

// acc += sum of val(e) * in[col[e], half] over the entries [e0, e1), in entry
// order; a chunk's columns and values are loaded before its rows.
template <typename Val>
__device__ __forceinline__ void half_row_sum(int e0, int e1, const int *__restrict__ col, Val val,
                                             const float *__restrict__ in, int half, float4 &acc) {
  constexpr int U = 4;
  const float4 *__restrict__ in4 = reinterpret_cast<const float4 *>(in);
  for (int e = e0; e < e1; e += U) {
    int c[U];
    float a[U];
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int eu = min(e + u, e1 - 1);
      c[u] = col[eu];
      a[u] = val(eu);
    }
#pragma unroll
    for (int u = 0; u < U; u++) v[u] = in4[(size_t)c[u] * (S / 4) + half];
#pragma unroll
    for (int u = 0; u < U; u++)
      if (e + u < e1) {
        acc.x = fmaf(a[u], v[u].x, acc.x);
        acc.y = fmaf(a[u], v[u].y, acc.y);
        acc.z = fmaf(a[u], v[u].z, acc.z);
        acc.w = fmaf(a[u], v[u].w, acc.w);
      }
  }
}

// f(i, half) over the nodes, two neighbouring lanes per node.
template <typename F>
__device__ __forceinline__ void half_rows(int N, F f) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < 2ll * N;
       t += (long long)gridDim.x * blockDim.x)
    f((int)(t >> 1), (int)(t & 1));
}

// OUT = M IN for an S-column block, M in CRS.
__global__ void __launch_bounds__(kThreads)
    k_spmm8(int N, const int *__restrict__ rp, const int *__restrict__ col,
            const float *__restrict__ val, const float *__restrict__ in,
            float *__restrict__ out) {
  half_rows(N, [&](int i, int half) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    half_row_sum(rp[i], rp[i + 1], col, [&](int e) { return val[e]; }, in, half, acc);
    reinterpret_cast<float4 *>(out)[(size_t)i * (S / 4) + half] = acc;
  });
}

// One damped-Jacobi step on the Jacobi-scaled matrix for the columns [c0, c1):
// out = sc (in - om Ahat in); the other columns are copied. (sc is the column
// scale, applied in the last step.)
__global__ void __launch_bounds__(kThreads)
    k_smooth8(int N, const int *__restrict__ rp, const int *__restrict__ col,
              const float *__restrict__ val, float om, float sc, int c0, int c1,
              const float *__restrict__ in, float *__restrict__ out) {
  half_rows(N, [&](int i, int half) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    half_row_sum(rp[i], rp[i + 1], col, [&](int e) { return val[e]; }, in, half, t);
    float4 v = reinterpret_cast<const float4 *>(in)[(size_t)i * (S / 4) + half];
    const int c = 4 * half;
    v.x = c + 0 >= c0 && c + 0 < c1 ? sc * fmaf(-om, t.x, v.x) : v.x;
    v.y = c + 1 >= c0 && c + 1 < c1 ? sc * fmaf(-om, t.y, v.y) : v.y;
    v.z = c + 2 >= c0 && c + 2 < c1 ? sc * fmaf(-om, t.z, v.z) : v.z;
    v.w = c + 3 >= c0 && c + 3 < c1 ? sc * fmaf(-om, t.w, v.w) : v.w;
    reinterpret_cast<float4 *>(out)[(size_t)i * (S / 4) + half] = v;
  });
}

// T3 = G^T T2 (G^T rows with values ghat[t2g[t]]), R = T3 - V,
// rho = 2 R / (N S), partial sums of R^2 -> *loss (last CTA).
__global__ void __launch_bounds__(kThreads)
    k_loss_residual(int N, const int *__restrict__ tptr, const int *__restrict__ tcol,
                    const float *__restrict__ ghat, const int *__restrict__ t2g,
                    const float *__restrict__ T2, const float *__restrict__ V,
                    float *__restrict__ rho, double *partials, unsigned *ticket, float *loss) {
  const float scale = 2.f / ((float)N * S);
  double acc = 0.0;
  half_rows(N, [&](int i, int half) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    half_row_sum(tptr[i], tptr[i + 1], tcol, [&](int e) { return ghat[t2g[e]]; }, T2, half, t);
    const size_t at = (size_t)i * (S / 4) + half;
    const float4 v = reinterpret_cast<const float4 *>(V)[at];
    const float4 d = make_float4(t.x - v.x, t.y - v.y, t.z - v.z, t.w - v.w);
    acc += (double)d.x * d.x;
    acc += (double)d.y * d.y;
    acc += (double)d.z * d.z;
    acc += (double)d.w * d.w;
    reinterpret_cast<float4 *>(rho)[at] =
        make_float4(scale * d.x, scale * d.y, scale * d.z, scale * d.w);
  });
  double in[1] = {acc}, out[1];
  if (grid_reduce<1>(in, partials, ticket, out) && threadIdx.x == 0)
    *loss = (float)(out[0] / ((double)N * S));
}

__device__ __forceinline__ float dot4f(float4 a, float4 b, float s) {
  s = fmaf(a.x, b.x, s);
  s = fmaf(a.y, b.y, s);
  s = fmaf(a.z, b.z, s);
  return fmaf(a.w, b.w, s);
}

// Over row i of G, with dGhat_ij = sum_s T2[i,s] rho[j,s] + dT1[i,s] V[j,s]:
// the gradient w.r.t. the head outputs o_i = [a, dg, u, v] that row i has,
//   d dg_i = dGhat_ii sigmoid(dg_i + offset)
//   d a_i  = sum_{j<i} c_ij,  d u_i = sum_{j<i} c_ij v_j,  c_ij = dGhat_ij w_ij,
// and c_ij itself for k_grad_cols (diagonal entries have none).
__global__ void __launch_bounds__(kThreads)
    k_grad_rows(int N, const int *__restrict__ gptr, const int *__restrict__ gcol,
                const int *__restrict__ g2a, const float *__restrict__ ahat,
                const float *__restrict__ T2, const float *__restrict__ dT1,
                const float *__restrict__ rho, const float *__restrict__ V,
                const float *__restrict__ o, float *__restrict__ cfac,
                float *__restrict__ dO) {
  const unsigned pair = 3u << (threadIdx.x & 30);  // the two lanes of a row
  half_rows(N, [&](int i, int half) {
    const size_t at = (size_t)i * (S / 4) + half;
    const float4 t2 = reinterpret_cast<const float4 *>(T2)[at];
    const float4 d1 = reinterpret_cast<const float4 *>(dT1)[at];
    const float sg = sigmoid(o[(size_t)i * NOUT + 1] + DIAG_OFFSET);
    float da = 0.f, ddg = 0.f;
    float2 du = make_float2(0.f, 0.f);
    constexpr int U = 4;
    const int e1 = gptr[i + 1];
    for (int e = gptr[i]; e < e1; e += U) {
      int j[U];
      float w[U];
      float4 r[U], v[U];
      float2 vj[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int eu = min(e + u, e1 - 1);
        j[u] = gcol[eu];
        w[u] = fabsf(ahat[g2a[eu]]);
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        const size_t jt = (size_t)j[u] * (S / 4) + half;
        r[u] = reinterpret_cast<const float4 *>(rho)[jt];
        v[u] = reinterpret_cast<const float4 *>(V)[jt];
        vj[u] = reinterpret_cast<const float2 *>(o + (size_t)j[u] * NOUT + 2 + RANK)[half];
      }
#pragma unroll
      for (int u = 0; u < U; u++)
        if (e + u < e1) {
          float s = dot4f(t2, r[u], dot4f(d1, v[u], 0.f));
          s += __shfl_xor_sync(pair, s, 1);
          if (j[u] == i) {
            ddg += s * sg;
          } else {
            const float c = s * w[u];
            da += c;
            du.x = fmaf(c, vj[u].x, du.x);
            du.y = fmaf(c, vj[u].y, du.y);
            if (half == 0) cfac[e + u] = c;
          }
        }
    }
    float *d = dO + (size_t)i * NOUT;
    if (half == 0) reinterpret_cast<float2 *>(d)[0] = make_float2(da, ddg);
    reinterpret_cast<float2 *>(d + 2)[half] = du;
  });
}

// d v_i = sum_{r>i} c_ri u_r over row i of G^T.
__global__ void __launch_bounds__(kThreads)
    k_grad_cols(int N, const int *__restrict__ tptr, const int *__restrict__ tcol,
                const int *__restrict__ t2g, const float *__restrict__ cfac,
                const float *__restrict__ o, float *__restrict__ dO) {
  half_rows(N, [&](int i, int half) {
    float2 dv = make_float2(0.f, 0.f);
    constexpr int U = 4;
    const int t1 = tptr[i + 1];
    for (int t = tptr[i]; t < t1; t += U) {
      int r[U];
      float c[U];
      float2 ur[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int tu = min(t + u, t1 - 1);
        r[u] = tcol[tu];
        c[u] = cfac[t2g[tu]];  // unused on the diagonal
      }
#pragma unroll
      for (int u = 0; u < U; u++)
        ur[u] = reinterpret_cast<const float2 *>(o + (size_t)r[u] * NOUT + 2)[half];
#pragma unroll
      for (int u = 0; u < U; u++)
        if (t + u < t1 && r[u] != i) {
          dv.x = fmaf(c[u], ur[u].x, dv.x);
          dv.y = fmaf(c[u], ur[u].y, dv.y);
        }
    }
    reinterpret_cast<float2 *>(dO + (size_t)i * NOUT + 2 + RANK)[half] = dv;
  });
}

// --- the layers --------------------------------------------------------------

// dh of node i, features 4 q .. 4 q + 3: dself_i + sum_{j != i} |Ahat_ij| dagg_j
// in entry order (the aggregation weights are symmetric), what the layer above
// left for its input. index and ahat point to the node's entries.
__device__ __forceinline__ float4 gather_dh(int i, int q, int entries, const int *index,
                                            const float *ahat, const float *__restrict__ dself,
                                            const float *__restrict__ dagg) {
  constexpr int U = 8;
  const float4 *__restrict__ in = reinterpret_cast<const float4 *>(dagg);
  float4 s = reinterpret_cast<const float4 *>(dself)[(size_t)i * (W / 4) + q];
  for (int e = 0; e < entries; e += U) {
    int c[U];
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      c[u] = index[min(e + u, entries - 1)];
      v[u] = in[(size_t)c[u] * (W / 4) + q];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const float w = fabsf(ahat[min(e + u, entries - 1)]);
      if (e + u < entries && c[u] != i) {
        s.x = fmaf(w, v[u].x, s.x);
        s.y = fmaf(w, v[u].y, s.y);
        s.z = fmaf(w, v[u].z, s.z);
        s.w = fmaf(w, v[u].w, s.w);
      }
    }
  }
  return s;
}

__device__ __forceinline__ float4 masked(float4 v, uint32_t m) {
  return make_float4(m & 1u ? v.x : 0.f, m & 2u ? v.y : 0.f, m & 4u ? v.z : 0.f,
                     m & 8u ? v.w : 0.f);
}

// v as a sum of three BF16 values, largest first (24 bits: exact but for values
// whose last bits fall below the smallest FP32 numbers). Above BF16's largest number
// the first term is rounded towards zero; an infinite v is its first term alone, as
// the difference would be NaN.
__device__ __forceinline__ void split3(float v, __nv_bfloat16 (&s)[3]) {
  s[0] = __float2bfloat16_rn(v);
  float rest = v - __bfloat162float(s[0]);
  if (fabsf(__bfloat162float(s[0])) > 3.4e38f) {  // infinite
    s[0] = __float2bfloat16_rz(v);
    rest = fabsf(v) > FLT_MAX ? 0.f : v - __bfloat162float(s[0]);
  }
  s[1] = __float2bfloat16_rn(rest);
  s[2] = __float2bfloat16_rn(rest - __bfloat162float(s[1]));
}

// Four 8 x 8 matrices of 16-bit elements from shared memory, lane l giving the
// address of row l % 8 of matrix l / 8; transposed, each register holds the
// matrix's columns.
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const void *p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p))
               : "memory");
}
__device__ __forceinline__ void ldmatrix4_t(uint32_t (&r)[4], const void *p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p))
               : "memory");
}

// 16 bytes from global to shared memory, asynchronously; zeros if !in.
__device__ __forceinline__ void copy16_async(void *dst, const void *src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
               :
               : "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0)
               : "memory");
}

__device__ __forceinline__ void copy4_async(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;"
               :
               : "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
// Until at most NEWER of this thread's groups are in flight.
template <int NEWER>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" : : "n"(NEWER) : "memory");
}

constexpr int kBackWarps = 4;   // warps per CTA
constexpr int kBackCtas = 3;    // CTAs per SM
constexpr int kBackNodes = 16;  // nodes of a warp's step
constexpr int kBackEntries = 224;  // entries of a step held in shared memory

// Backward through layer `layer`, a step of 16 nodes per warp:
//   dh    HEAD (the last layer): W_h^T dO;  else gather_dh of the layer above
//   dpre  = dh * [pre > 0]
//   dself = dh + (W_l^T dpre)[0:W],  dagg = (W_l^T dpre)[W:2W]   (W_l in BF16)
//   and this CTA's sums of dpre [h ; agg]^T and dpre (and with HEAD of dO h^T and
//   dO), into its row of `partial`, in parameter layout.
// Both products have one operand in BF16 (W_l, and h and agg); the other, dpre,
// is FP32 and enters the tensor cores as three BF16 terms (split3), smallest
// first, so that every product is exact and FP32 sums are what is rounded.
// Against 64-bit arithmetic with the same BF16 rounding points the whole
// gradient is off by 1.6e-7 to 2.4e-6 (2-norm, 7- and 27-point grids and graphs),
// with FP32 multiply-adds 4.2e-7 to 2.3e-6.
// What bounds it is latency (DRAM and L2 round trips at 12 warps per SM, whose
// sums take 64 registers): so the next step's row pointers and entries, or dO,
// and this step's h and agg are fetched ahead. us a layer at 96^3 (885k nodes,
// 70 for its bytes at the measured 6.54 TB/s): one pass per product on FP32
// multiply-adds 1430; multiply-adds in registers, one pass 624 (last layer 456); tensor
// cores 320 (297); fetching ahead 259 (202).
template <bool HEAD>
__global__ void __launch_bounds__(32 * kBackWarps, kBackCtas)
    k_layer_back(int N, const int *__restrict__ ptr, const int *__restrict__ index,
                 const float *__restrict__ ahat, const float *__restrict__ P, int layer,
                 const float *__restrict__ dO, const __nv_bfloat16 *__restrict__ hout,
                 const float *__restrict__ dself_in, const float *__restrict__ dagg_in,
                 const uint32_t *__restrict__ mask, const __nv_bfloat16 *__restrict__ hin,
                 const __nv_bfloat16 *__restrict__ agg, float *__restrict__ dself,
                 float *__restrict__ dagg, float *__restrict__ partial) {
  constexpr int M = kBackNodes;
  // Row lengths that spread the 8 rows of a fragment over the banks.
  struct __align__(16) Step {
    float dh[M][W + 8];
    __nv_bfloat16 dp[3][M][W + 8];
    __nv_bfloat16 x[M][2 * W + 8];
    int col[HEAD ? 1 : kBackEntries];
    float w[HEAD ? 1 : kBackEntries];
  };
  constexpr int kLayerSums = 2 * W * W + W, kHeadSums = NOUT * W + NOUT;
  constexpr int kSums = kLayerSums + (HEAD ? kHeadSums : 0);
  static_assert(sizeof(Step) % 16 == 0 && sizeof(float) * kSums <= sizeof(Step) * kBackWarps,
                "k_layer_back");
  __shared__ __align__(16) Step sh[kBackWarps];
  __shared__ __align__(16) __nv_bfloat16 sW[W][2 * W + 8];
  __shared__ __align__(16) float sO[HEAD ? kBackWarps : 1][HEAD ? M * NOUT : 1];
  const int warp = threadIdx.x >> 5, f = threadIdx.x & 31;
  const float *Wl = P + OFF_L0 + layer * L_STRIDE;
  for (int t = threadIdx.x; t < W * 2 * W; t += blockDim.x)
    sW[t / (2 * W)][t % (2 * W)] = __float2bfloat16_rn(Wl[t]);
  __syncthreads();
  float gw[2][8][4] = {};           // dW: 16-row and 8-column tiles
  float4 gb4 = make_float4(0.f, 0.f, 0.f, 0.f);
  float gb = 0.f, wh[HEAD ? NOUT : 1], gh[HEAD ? NOUT : 1], ghb = 0.f;
#pragma unroll
  for (int k = 0; k < (HEAD ? NOUT : 1); k++) {
    wh[k] = HEAD ? P[OFF_WH + k * W + f] : 0.f;
    gh[k] = 0.f;
  }
  // Fragment addresses: row f % 8 (+ 8) and column 0 or 8 by the quarter warp.
  const int r8 = f & 7, lo = (f >> 3) & 1, hi = f >> 4;

  Step &st = sh[warp];
  const int steps = (N + M - 1) / M, stride = gridDim.x * kBackWarps;
  int g = blockIdx.x * kBackWarps + warp;
  // What the next step begins with is fetched during this one: dO, or the row
  // pointers (lane r: node r's first entry, lane 16: the end), and the entries
  // if they fit.
  constexpr int kOd = M * NOUT / 32;
  float od[HEAD ? kOd : 1];
  int row = 0;
  auto fetch_rows = [&](int s0) {
    if constexpr (HEAD) {
#pragma unroll
      for (int k = 0; k < kOd; k++) {
        const size_t at = (size_t)s0 * M * NOUT + f + 32 * k, end = (size_t)N * NOUT;
        od[k] = dO[at < end ? at : end - 1];
      }
    } else {
      row = ptr[min((long long)s0 * M + min(f, M), (long long)N)];
    }
  };
  auto fetch_entries = [&]() {
    if constexpr (!HEAD) {
      const int e0 = __shfl_sync(0xffffffffu, row, 0);
      const int n = __shfl_sync(0xffffffffu, row, M) - e0;
      if (n <= kBackEntries)
        for (int t = f; t < n; t += 32) {
          copy4_async(&st.col[t], index + e0 + t);
          copy4_async(&st.w[t], ahat + e0 + t);
        }
    }
    copy_commit();
  };
  if (g < steps) {
    fetch_rows(g);
    fetch_entries();
  }
  for (; g < steps; g += stride) {
    const int base = g * M;
    __syncwarp();  // the last step's reads are done
    const uint32_t mine = mask[min(base + f % M, N - 1)];
    // h and agg of the step: two 16-byte pieces each per lane, copied while dh
    // is formed (rows past the last are zero-filled).
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int r = (f >> 2) + 8 * u;
      const bool in = base + r < N;
      const size_t at = (size_t)(in ? base + r : 0) * (W / 8) + (f & 3);
      copy16_async(&st.x[r][8 * (f & 3)], reinterpret_cast<const uint4 *>(hin) + at, in);
      copy16_async(&st.x[r][W + 8 * (f & 3)], reinterpret_cast<const uint4 *>(agg) + at, in);
    }
    copy_commit();
    if constexpr (HEAD) {
      __nv_bfloat16 hv[M];
#pragma unroll
      for (int r = 0; r < M; r++) hv[r] = hout[(size_t)min(base + r, N - 1) * W + f];
#pragma unroll
      for (int k = 0; k < kOd; k++)
        sO[warp][f + 32 * k] =
            (size_t)base * NOUT + f + 32 * k < (size_t)N * NOUT ? od[k] : 0.f;
      __syncwarp();
      fetch_rows(g + stride);
#pragma unroll
      for (int r = 0; r < M; r++) {
        const float h3 = __bfloat162float(hv[r]);
        const uint32_t m = __shfl_sync(0xffffffffu, mine, r);
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < NOUT; k += 2) {
          const float2 d = *reinterpret_cast<const float2 *>(&sO[warp][r * NOUT + k]);
          s = fmaf(wh[k], d.x, s);
          s = fmaf(wh[k + 1], d.y, s);
          gh[k] = fmaf(d.x, h3, gh[k]);
          gh[k + 1] = fmaf(d.y, h3, gh[k + 1]);
        }
        if (f < NOUT) ghb += sO[warp][r * NOUT + f];
        const float dp = (m >> f) & 1u ? s : 0.f;
        gb += dp;
        __nv_bfloat16 t[3];
        split3(dp, t);
        st.dh[r][f] = s;
#pragma unroll
        for (int k = 0; k < 3; k++) st.dp[k][r][f] = t[k];
      }
    } else {
      const int q = f & 7, e0 = __shfl_sync(0xffffffffu, row, 0);
      const bool held = __shfl_sync(0xffffffffu, row, M) - e0 <= kBackEntries;
      copy_wait<1>();
      __syncwarp();
      // Generic pointers: the entries are in shared or in global memory.
      const int *cp = held ? st.col : index + e0;
      const float *wp = held ? st.w : ahat + e0;
#pragma unroll 1
      for (int k = 0; k < M / 4; k++) {
        const int r = 4 * k + (f >> 3), i = base + r;
        const int j0 = __shfl_sync(0xffffffffu, row, r), j1 = __shfl_sync(0xffffffffu, row, r + 1);
        const uint32_t m = __shfl_sync(0xffffffffu, mine, r);
        float4 dh = make_float4(0.f, 0.f, 0.f, 0.f), dp = dh;
        if (i < N) {
          dh = gather_dh(i, q, j1 - j0, cp + (j0 - e0), wp + (j0 - e0), dself_in, dagg_in);
          dp = masked(dh, m >> (4 * q));
        }
        gb4.x += dp.x;
        gb4.y += dp.y;
        gb4.z += dp.z;
        gb4.w += dp.w;
        __nv_bfloat16 t[4][3];
        split3(dp.x, t[0]);
        split3(dp.y, t[1]);
        split3(dp.z, t[2]);
        split3(dp.w, t[3]);
        *reinterpret_cast<float4 *>(&st.dh[r][4 * q]) = dh;
#pragma unroll
        for (int u = 0; u < 3; u++)
          *reinterpret_cast<uint2 *>(&st.dp[u][r][4 * q]) =
              make_uint2(pack2(t[0][u], t[1][u]), pack2(t[2][u], t[3][u]));
      }
      fetch_rows(g + stride);
    }
    copy_wait<0>();
    __syncwarp();
    // dW += dpre^T [h ; agg]: 32 x 64 over the step's 16 nodes.
    {
      uint32_t b[4][4];
#pragma unroll
      for (int t = 0; t < 4; t++) ldmatrix4_t(b[t], &st.x[r8 + 8 * lo][16 * t + 8 * hi]);
#pragma unroll
      for (int u = 2; u >= 0; u--)
#pragma unroll
        for (int mt = 0; mt < 2; mt++) {
          uint32_t a[4];
          ldmatrix4_t(a, &st.dp[u][r8 + 8 * hi][16 * mt + 8 * lo]);
#pragma unroll
          for (int t = 0; t < 4; t++) {
            const uint32_t b0[2] = {b[t][0], b[t][1]}, b1[2] = {b[t][2], b[t][3]};
            mma_bf16_16816(gw[mt][2 * t], a, b0);
            mma_bf16_16816(gw[mt][2 * t + 1], a, b1);
          }
        }
    }
    if (g + stride < steps) fetch_entries();
    // dX = dpre W_l: 16 x 64, first the half of h, then that of agg.
    uint32_t a[3][2][4];
#pragma unroll
    for (int u = 0; u < 3; u++)
#pragma unroll
      for (int ks = 0; ks < 2; ks++)
        ldmatrix4(a[u][ks], &st.dp[u][r8 + 8 * lo][16 * ks + 8 * hi]);
#pragma unroll
    for (int half = 0; half < 2; half++) {
      float acc[4][4] = {};
#pragma unroll
      for (int t = 0; t < 2; t++) {
        uint32_t b[2][4];
#pragma unroll
        for (int ks = 0; ks < 2; ks++)
          ldmatrix4_t(b[ks], &sW[16 * ks + r8 + 8 * lo][W * half + 16 * t + 8 * hi]);
#pragma unroll
        for (int u = 2; u >= 0; u--)
#pragma unroll
          for (int ks = 0; ks < 2; ks++) {
            const uint32_t b0[2] = {b[ks][0], b[ks][1]}, b1[2] = {b[ks][2], b[ks][3]};
            mma_bf16_16816(acc[2 * t], a[u][ks], b0);
            mma_bf16_16816(acc[2 * t + 1], a[u][ks], b1);
          }
      }
      float *out = half ? dagg : dself;
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int r = (f >> 2) + 8 * k;
        if (base + r >= N) continue;
#pragma unroll
        for (int nt = 0; nt < 4; nt++) {
          const int c = 8 * nt + 2 * (f & 3);
          float2 v = make_float2(acc[nt][2 * k], acc[nt][2 * k + 1]);
          if (half == 0) {
            const float2 d = *reinterpret_cast<const float2 *>(&st.dh[r][c]);
            v = make_float2(d.x + v.x, d.y + v.y);
          }
          *reinterpret_cast<float2 *>(&out[(size_t)(base + r) * W + c]) = v;
        }
      }
    }
  }
  // The CTA's sums, warp after warp.
  if (!HEAD) {
    float v[4] = {gb4.x, gb4.y, gb4.z, gb4.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      v[k] += __shfl_xor_sync(0xffffffffu, v[k], 8);
      v[k] += __shfl_xor_sync(0xffffffffu, v[k], 16);
    }
    gb4 = make_float4(v[0], v[1], v[2], v[3]);
  }
  float *sum = reinterpret_cast<float *>(sh);
  __syncthreads();
  for (int w = 0; w < kBackWarps; w++) {
    auto put = [&](int at, float v) { sum[at] = w ? sum[at] + v : v; };
    if (warp == w) {
#pragma unroll
      for (int mt = 0; mt < 2; mt++)
#pragma unroll
        for (int nt = 0; nt < 8; nt++)
#pragma unroll
          for (int k = 0; k < 4; k++)
            put((16 * mt + (f >> 2) + 8 * (k >> 1)) * 2 * W + 8 * nt + 2 * (f & 3) + (k & 1),
                gw[mt][nt][k]);
      if constexpr (HEAD) {
        put(2 * W * W + f, gb);
#pragma unroll
        for (int k = 0; k < NOUT; k++) put(kLayerSums + k * W + f, gh[k]);
        if (f < NOUT) put(kLayerSums + NOUT * W + f, ghb);
      } else if (f < 8) {
        put(2 * W * W + 4 * f, gb4.x);
        put(2 * W * W + 4 * f + 1, gb4.y);
        put(2 * W * W + 4 * f + 2, gb4.z);
        put(2 * W * W + 4 * f + 3, gb4.w);
      }
    }
    __syncthreads();
  }
  float *out = partial + (size_t)blockIdx.x * NPARAMS + OFF_L0 + layer * L_STRIDE;
  for (int t = threadIdx.x; t < kSums; t += blockDim.x) out[t] = sum[t];
}
static_assert(OFF_WH == OFF_L0 + 3 * L_STRIDE && OFF_BH == OFF_WH + NOUT * W,
              "the head's parameters follow the last layer's");

// Embedding: this CTA's sums of dpre0 f^T and dpre0, dpre0 = gather_dh * [pre0 >
// 0]; eight lanes a node. Bound by the gathered rows (128 bytes an entry): 157 us
// at 96^3, where the gather, the mask and the sums took 355 as passes of their own.
constexpr int kEmbedBackThreads = 256;
__global__ void __launch_bounds__(kEmbedBackThreads)
    k_embed_back(int N, const int *__restrict__ ptr, const int *__restrict__ index,
                 const float *__restrict__ ahat, const float *__restrict__ dself,
                 const float *__restrict__ dagg, const uint32_t *__restrict__ mask,
                 const float *__restrict__ feat, float *__restrict__ partial) {
  constexpr int kW = kEmbedBackThreads / 32, kSums = W * NIN + W;
  __shared__ float sum[kW][kSums];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 7;
  float acc[4][NIN + 1] = {};
  const int per = kW * 4;
  for (int i = (blockIdx.x * kW + warp) * 4 + (lane >> 3); i < N; i += gridDim.x * per) {
    const float4 d4 =
        masked(gather_dh(i, q, ptr[i + 1] - ptr[i], index + ptr[i], ahat + ptr[i], dself, dagg),
               mask[i] >> (4 * q));
    const float4 f4 = reinterpret_cast<const float4 *>(feat)[i];
    const float d[4] = {d4.x, d4.y, d4.z, d4.w}, x[NIN] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
    for (int a = 0; a < 4; a++) {
#pragma unroll
      for (int k = 0; k < NIN; k++) acc[a][k] = fmaf(d[a], x[k], acc[a][k]);
      acc[a][NIN] += d[a];
    }
  }
  __syncwarp();
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int k = 0; k <= NIN; k++) {
      float v = acc[a][k];
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 16);
      if (lane < 8) sum[warp][k < NIN ? (4 * q + a) * NIN + k : W * NIN + 4 * q + a] = v;
    }
  __syncthreads();
  float *out = partial + (size_t)blockIdx.x * NPARAMS + OFF_WIN;
  for (int t = threadIdx.x; t < kSums; t += blockDim.x) {
    float v = sum[0][t];
    for (int w = 1; w < kW; w++) v += sum[w][t];
    out[t] = v;
  }
}
static_assert(OFF_BIN == OFF_WIN + W * NIN && NIN == 4, "the embedding's parameters");

// out[k] = sum over the CTAs of partial[cta][k], in a fixed order: 32
// parameters per CTA, eight warps over the rows.
__global__ void __launch_bounds__(kThreads)
    k_sum_partials(int rows, const float *__restrict__ partial, float *__restrict__ out) {
  __shared__ float sh[kWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (k < NPARAMS) {
#pragma unroll 8
    for (int c = warp; c < rows; c += kWarps) s += partial[(size_t)c * NPARAMS + k];
  }
  sh[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && k < NPARAMS) {
    for (int w = 1; w < kWarps; w++) s += sh[w][lane];
    out[k] = s;
  }
}

}  // namespace learned
}  // namespace cgx

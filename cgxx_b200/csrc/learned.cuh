// Learned preconditioner M^-1 = G G^T + eps D^-1 (no counterpart in the
// reference): device kernels for
//   - the Jacobi-scaled graph of A: 1/sqrt(A_ii), |Ahat_ij|, node features,
//     the pattern of G (lower triangle of A, diagonal included, storage
//     order) and of G^T (upper triangle), and the maps between them;
//   - the message-passing network that emits G's values (forward on BF16
//     tensor cores, mma.sync m16n8k16, FP32 accumulation);
//   - Adam and the training probes (the loss and the backward pass: train.cuh).
// The exact arithmetic is stated in oracle/gnn_oracle.py, the CPU oracle the
// tests compare these kernels with.
#pragma once

#include <cuda_bf16.h>

#include "device.cuh"

namespace cgx {
namespace learned {

constexpr int W = 32;       // feature width
constexpr int RANK = 4;     // rank of the off-diagonal bilinear term
constexpr int NIN = 4;      // node input features
constexpr int NOUT = 2 + 2 * RANK;
constexpr float DIAG_OFFSET = 0.5413f;
constexpr int S = 8;        // Hutchinson probe columns per training step

// Flat parameter layout (FP32), identical to oracle/gnn_oracle.py.
constexpr int OFF_WIN = 0;
constexpr int OFF_BIN = OFF_WIN + W * NIN;
constexpr int OFF_L0 = OFF_BIN + W;
constexpr int L_STRIDE = W * 2 * W + W;  // W_l then b_l
constexpr int OFF_WH = OFF_L0 + 3 * L_STRIDE;
constexpr int OFF_BH = OFF_WH + NOUT * W;
constexpr int NPARAMS = OFF_BH + NOUT;

__device__ __forceinline__ float softplus(float x) {
  return x > 20.f ? x : log1pf(expf(x));
}
__device__ __forceinline__ float sigmoid(float x) {
  return 1.f / (1.f + expf(-x));
}

// ---------------------------------------------------------------------------
// Scaled graph

// dis_i = 1 / sqrt(A_ii) (last diagonal entry of the row; 0 if none -> the
// set-up reports an error).
__global__ void k_inv_sqrt_diag(int N, const int *__restrict__ ptr,
                                const int *__restrict__ index,
                                const double *__restrict__ value,
                                double *dis, int *flag) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += gridDim.x * blockDim.x) {
    const int j = last_entry(index, ptr[i], ptr[i + 1], i);
    const double d = j >= 0 ? value[j] : 0.0;
    if (!(d > 0.0)) {
      atomicOr(flag, 1);
      dis[i] = 0.0;
    } else {
      dis[i] = 1.0 / sqrt(d);
    }
  }
}

// Ahat entries (FP32), node features and the lower/upper counts per row.
__global__ void k_scaled_rows(int N, const int *__restrict__ ptr,
                              const int *__restrict__ index,
                              const double *__restrict__ value,
                              const double *__restrict__ dis,
                              float *__restrict__ ahat, float *__restrict__ feat,
                              int *__restrict__ nlow, int *__restrict__ nup) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += gridDim.x * blockDim.x) {
    const double di = dis[i];
    float s = 0.f, mx = 0.f;
    int deg = 0, lo = 0, up = 0;
    constexpr int U = 4;
    const int j1 = ptr[i + 1];
    for (int j = ptr[i]; j < j1; j += U) {
      // Unconditional loads, a chunk's columns and values before its scales.
      int c[U];
      double v[U], dj[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        c[u] = index[min(j + u, j1 - 1)];
        v[u] = value[min(j + u, j1 - 1)];
      }
#pragma unroll
      for (int u = 0; u < U; u++) dj[u] = dis[c[u]];
#pragma unroll
      for (int u = 0; u < U; u++)
        if (j + u < j1) {
          const float a = (float)(v[u] * di * dj[u]);
          ahat[j + u] = a;
          if (c[u] != i) {
            s += fabsf(a);
            mx = fmaxf(mx, fabsf(a));
            deg++;
          }
          lo += c[u] <= i;
          up += c[u] >= i;
        }
    }
    feat[i * NIN + 0] = 1.f;
    feat[i * NIN + 1] = s;
    feat[i * NIN + 2] = (float)deg / 6.f;
    feat[i * NIN + 3] = mx;
    nlow[i] = lo;
    nup[i] = up;
  }
}

// Block-level exclusive scan helpers for the pattern build: three launches
// (per-block totals, scan of the totals, add offsets), out[0] = 0 and
// out[n] = total.
constexpr int kScanBlock = 1024;

__global__ void k_scan_blocks(int n, const int *__restrict__ in,
                              int *__restrict__ out, int *__restrict__ sums) {
  __shared__ int sh[kScanBlock];
  const int i = blockIdx.x * kScanBlock + threadIdx.x;
  sh[threadIdx.x] = i < n ? in[i] : 0;
  __syncthreads();
  for (int o = 1; o < kScanBlock; o <<= 1) {
    int v = threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
    __syncthreads();
    sh[threadIdx.x] += v;
    __syncthreads();
  }
  if (i < n) out[i + 1] = sh[threadIdx.x];  // inclusive, shifted by one
  if (threadIdx.x == kScanBlock - 1) sums[blockIdx.x] = sh[threadIdx.x];
}

__global__ void k_scan_sums(int nb, int *sums) {
  // One block; nb may exceed the block size: serial carry over chunks.
  __shared__ int sh[kScanBlock];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < nb; base += kScanBlock) {
    const int i = base + threadIdx.x;
    sh[threadIdx.x] = i < nb ? sums[i] : 0;
    __syncthreads();
    for (int o = 1; o < kScanBlock; o <<= 1) {
      int v = threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
      __syncthreads();
      sh[threadIdx.x] += v;
      __syncthreads();
    }
    const int excl = carry + sh[threadIdx.x] - (i < nb ? sums[i] : 0);
    __syncthreads();
    if (i < nb) sums[i] = excl;  // exclusive block offsets
    if (threadIdx.x == kScanBlock - 1) carry += sh[kScanBlock - 1];
    __syncthreads();
  }
}

__global__ void k_scan_add(int n, int *__restrict__ out,
                           const int *__restrict__ sums) {
  const int i = blockIdx.x * kScanBlock + threadIdx.x;
  if (i < n) out[i + 1] += sums[blockIdx.x];
  if (i == 0) out[0] = 0;
}

// Fills the G (lower) and G^T (upper) patterns in A's storage order, and for
// each G entry the position of the same entry in A (g2a).
__global__ void k_fill_patterns(int N, const int *__restrict__ ptr,
                                const int *__restrict__ index,
                                const int *__restrict__ gptr,
                                const int *__restrict__ tptr,
                                int *__restrict__ gcol, int *__restrict__ grow,
                                int *__restrict__ tcol,
                                int *__restrict__ g2a) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += gridDim.x * blockDim.x) {
    int g = gptr[i], t = tptr[i];
    for (int j = ptr[i]; j < ptr[i + 1]; j++) {
      const int c = index[j];
      if (c <= i) {
        gcol[g] = c;
        grow[g] = i;
        g2a[g++] = j;
      }
      if (c >= i) tcol[t++] = c;
    }
  }
}

// For every G entry (i, j): its position in G^T row j (entry with column i),
// found by scanning that row. A missing mirror entry (pattern not symmetric)
// sets the flag.
__global__ void k_transpose_map(int nnzL, const int *__restrict__ grow,
                                const int *__restrict__ gcol,
                                const int *__restrict__ tptr,
                                const int *__restrict__ tcol,
                                int *__restrict__ g2t, int *__restrict__ t2g,
                                int *flag) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nnzL;
       e += gridDim.x * blockDim.x) {
    const int i = grow[e], j = gcol[e];
    int pos = -1;
    for (int k = tptr[j]; k < tptr[j + 1]; k++)
      if (tcol[k] == i) {
        pos = k;
        break;
      }
    g2t[e] = pos;
    if (pos < 0)
      atomicOr(flag, 2);
    else
      t2g[pos] = e;
  }
}

// ---------------------------------------------------------------------------
// Network forward

__device__ __forceinline__ float relu(float x) { return x > 0.f ? x : 0.f; }

// h0 = bf16(relu(W_in f + b_in)). For the backward pass: bit f of mask[i] says
// that pre-activation f of node i is positive, which is all that it reads of
// them (4 bytes per node and layer instead of 128).
__global__ void k_embed(int N, const float *__restrict__ feat,
                        const float *__restrict__ P, __nv_bfloat16 *__restrict__ h,
                        uint32_t *__restrict__ mask) {
  // One thread per node: W_in and b_in (contiguous in P) from shared memory,
  // the node's 4 features in one 16-byte load, its 32 outputs in four
  // 16-byte stores.
  __shared__ float sW[W * NIN + W];
  for (int t = threadIdx.x; t < W * NIN + W; t += blockDim.x) sW[t] = P[OFF_WIN + t];
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += gridDim.x * blockDim.x) {
    const float4 f4 = *reinterpret_cast<const float4 *>(feat + (size_t)i * NIN);
    const float fv[NIN] = {f4.x, f4.y, f4.z, f4.w};
    uint4 out[W / 8];
    __nv_bfloat16 *ob = reinterpret_cast<__nv_bfloat16 *>(out);
    uint32_t bits = 0u;
#pragma unroll
    for (int f = 0; f < W; f++) {
      float s = sW[W * NIN + f];
#pragma unroll
      for (int k = 0; k < NIN; k++) s = fmaf(sW[f * NIN + k], fv[k], s);
      bits |= s > 0.f ? 1u << f : 0u;
      ob[f] = __float2bfloat16_rn(relu(s));
    }
    if (mask) mask[i] = bits;
    uint4 *dst = reinterpret_cast<uint4 *>(h + (size_t)i * W);
#pragma unroll
    for (int q = 0; q < W / 8; q++) dst[q] = out[q];
  }
}

// Packs two bf16 values into the 32-bit register layout of an mma operand.
__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) |
         ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4],
                                               const uint32_t (&a)[4],
                                               const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// One message-passing layer. A warp owns 16 nodes: it gathers
// agg_i = sum_{j != i} |Ahat_ij| h_j (lane f accumulates feature f, FP32),
// stages X = [h_i ; bf16(agg_i)] (16 x 64, BF16) in shared memory, multiplies
// by W_l^T on the tensor cores (4 k-steps x 4 n-tiles of m16n8k16, FP32
// accumulators), adds the bias and writes h_i + relu(pre) as BF16.
//
// HEAD (the last layer): also the head outputs o_i = W_h h_i + b_h (FP32), two
// lanes a node with five outputs each, from the staged rows; h itself is stored
// only if hout is given (the backward pass reads it). At 96^3 the layer takes 108
// us with the head, against 89 and 54 for the layer and a pass of its own over h.
constexpr int kLayerWarps = 8;
// Chunks of four neighbours at 4 CTAs per SM; eight at 3 (2) CTAs: 96^3 86 -> 92
// (106) us, 2M-point graph 331 -> 375 (407).
template <bool HEAD>
__global__ void __launch_bounds__(32 * kLayerWarps, 4)
    k_layer(int N, const int *__restrict__ ptr, const int *__restrict__ index,
            const float *__restrict__ ahat, const float *__restrict__ P,
            int layer, const __nv_bfloat16 *__restrict__ hin,
            __nv_bfloat16 *__restrict__ hout, __nv_bfloat16 *__restrict__ agg_out,
            uint32_t *__restrict__ mask_out, float *__restrict__ o) {
  __shared__ __align__(16) __nv_bfloat16 sW[W][2 * W + 8];  // W_l[n][k], rows padded (banks)
  __shared__ __align__(16) __nv_bfloat16 sX[kLayerWarps][16][2 * W + 8];  // padded rows
  __shared__ float sB[W];
  __shared__ __align__(16) float sWh[HEAD ? NOUT : 1][W + 4];  // padded rows (banks)
  __shared__ float sBh[NOUT];
  const float *Wl = P + OFF_L0 + layer * L_STRIDE;
  for (int t = threadIdx.x; t < W * 2 * W; t += blockDim.x)
    sW[t / (2 * W)][t % (2 * W)] = __float2bfloat16_rn(Wl[t]);
  for (int t = threadIdx.x; t < W; t += blockDim.x) sB[t] = Wl[W * 2 * W + t];
  if constexpr (HEAD) {
    for (int t = threadIdx.x; t < NOUT * W; t += blockDim.x) sWh[t / W][t % W] = P[OFF_WH + t];
    for (int t = threadIdx.x; t < NOUT; t += blockDim.x) sBh[t] = P[OFF_BH + t];
  }
  __syncthreads();

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, tq = lane & 3;
  const int groups = (N + 15) / 16;
  for (int grp = blockIdx.x * kLayerWarps + warp; grp < groups;
       grp += gridDim.x * kLayerWarps) {
    const int base = grp * 16;
    // Gather: the warp's 16 nodes x 4 chunks of 8 features are 64 tasks,
    // two per lane, so all 16 nodes' neighbour rows are in flight at once;
    // a task reads 16 bytes (8 BF16 features) per neighbour, up to 4
    // neighbours requested before they are summed (in entry order).
    const uint4 *hin4 = reinterpret_cast<const uint4 *>(hin);
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int task = lane + 32 * q;
      const int r = task >> 2, c4 = task & 3;
      const int i = base + r;
      float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      uint4 own = make_uint4(0u, 0u, 0u, 0u);
      if (i < N) {
        own = hin4[(size_t)i * (W / 8) + c4];
        const int j0 = ptr[i], j1 = ptr[i + 1];
        for (int j = j0; j < j1; j += 4) {
          float w[4];
          uint4 hv[4];
          int cc[4];
          // All of a chunk's columns and weights first, then its
          // gathers: one round trip for each instead of one per entry. The
          // loads are unconditional (past the row's end: its last entry again,
          // weight 0), as a condition would make each a branch.
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int e = min(j + u, j1 - 1);
            cc[u] = index[e];
            w[u] = fabsf(ahat[e]);
          }
#pragma unroll
          for (int u = 0; u < 4; u++) hv[u] = hin4[(size_t)cc[u] * (W / 8) + c4];
#pragma unroll
          for (int u = 0; u < 4; u++) w[u] = cc[u] != i ? w[u] : 0.f;
#pragma unroll
          for (int u = 0; u < 4; u++) {
            if (j + u < j1) {
              const __nv_bfloat162 *b2 = reinterpret_cast<const __nv_bfloat162 *>(&hv[u]);
#pragma unroll
              for (int k = 0; k < 4; k++) {
                a[2 * k] = fmaf(w[u], __low2float(b2[k]), a[2 * k]);
                a[2 * k + 1] = fmaf(w[u], __high2float(b2[k]), a[2 * k + 1]);
              }
            }
          }
        }
      }
      uint4 ag;
      __nv_bfloat162 *ag2 = reinterpret_cast<__nv_bfloat162 *>(&ag);
#pragma unroll
      for (int k = 0; k < 4; k++) ag2[k] = __floats2bfloat162_rn(a[2 * k], a[2 * k + 1]);
      *reinterpret_cast<uint4 *>(&sX[warp][r][8 * c4]) = own;
      *reinterpret_cast<uint4 *>(&sX[warp][r][W + 8 * c4]) = ag;
      if (agg_out && i < N)
        reinterpret_cast<uint4 *>(agg_out)[(size_t)i * (W / 8) + c4] = ag;
    }
    __syncwarp();
    // pre = X W^T on the tensor cores.
    float acc[4][4];
#pragma unroll
    for (int nt = 0; nt < 4; nt++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[nt][q] = 0.f;
#pragma unroll
    for (int ks = 0; ks < 4; ks++) {
      const int k0 = ks * 16;
      uint32_t a[4];
      a[0] = pack2(sX[warp][g][k0 + 2 * tq], sX[warp][g][k0 + 2 * tq + 1]);
      a[1] = pack2(sX[warp][g + 8][k0 + 2 * tq], sX[warp][g + 8][k0 + 2 * tq + 1]);
      a[2] = pack2(sX[warp][g][k0 + 8 + 2 * tq], sX[warp][g][k0 + 8 + 2 * tq + 1]);
      a[3] = pack2(sX[warp][g + 8][k0 + 8 + 2 * tq],
                   sX[warp][g + 8][k0 + 8 + 2 * tq + 1]);
#pragma unroll
      for (int nt = 0; nt < 4; nt++) {
        const int n = nt * 8 + g;
        uint32_t b[2];
        b[0] = pack2(sW[n][k0 + 2 * tq], sW[n][k0 + 2 * tq + 1]);
        b[1] = pack2(sW[n][k0 + 8 + 2 * tq], sW[n][k0 + 8 + 2 * tq + 1]);
        mma_bf16_16816(acc[nt], a, b);
      }
    }
    // Epilogue: rows g and g+8, columns nt*8 + 2tq + {0,1}. The new h
    // replaces h_i in the staging rows (each element is read and written by
    // the lane that owns it), then the warp stores its 16 rows as 16-byte
    // chunks.
    uint32_t pos[2] = {0u, 0u};  // positive pre-activations of rows g, g + 8
#pragma unroll
    for (int nt = 0; nt < 4; nt++)
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int r = g + (q >= 2 ? 8 : 0);
        const int col = nt * 8 + 2 * tq + (q & 1);
        const float pre = acc[nt][q] + sB[col];
        pos[q >> 1] |= pre > 0.f ? 1u << col : 0u;
        const float hv = __bfloat162float(sX[warp][r][col]) + relu(pre);
        sX[warp][r][col] = __float2bfloat16_rn(hv);
      }
    if (mask_out) {
#pragma unroll
      for (int k = 0; k < 2; k++) {
        pos[k] |= __shfl_xor_sync(0xffffffffu, pos[k], 1);
        pos[k] |= __shfl_xor_sync(0xffffffffu, pos[k], 2);
        if (tq == 0 && base + g + 8 * k < N) mask_out[base + g + 8 * k] = pos[k];
      }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int task = lane + 32 * q;
      const int r = task >> 2, c4 = task & 3;
      if (base + r < N && (!HEAD || hout))
        reinterpret_cast<uint4 *>(hout)[(size_t)(base + r) * (W / 8) + c4] =
            *reinterpret_cast<const uint4 *>(&sX[warp][r][8 * c4]);
    }
    if constexpr (HEAD) {
      constexpr int K = NOUT / 2;
      const int r = lane & 15, k0 = (lane >> 4) * K;
      float s[K];
#pragma unroll
      for (int k = 0; k < K; k++) s[k] = sBh[k0 + k];
#pragma unroll
      for (int q = 0; q < W / 8; q++) {
        const uint4 raw = *reinterpret_cast<const uint4 *>(&sX[warp][r][8 * q]);
        const __nv_bfloat162 *b2 = reinterpret_cast<const __nv_bfloat162 *>(&raw);
#pragma unroll
        for (int hf = 0; hf < 2; hf++) {
          const float h0 = __low2float(b2[2 * hf]), h1 = __high2float(b2[2 * hf]);
          const float h2 = __low2float(b2[2 * hf + 1]), h3 = __high2float(b2[2 * hf + 1]);
#pragma unroll
          for (int k = 0; k < K; k++) {
            const float4 w = *reinterpret_cast<const float4 *>(&sWh[k0 + k][8 * q + 4 * hf]);
            s[k] = fmaf(w.x, h0, s[k]);
            s[k] = fmaf(w.y, h1, s[k]);
            s[k] = fmaf(w.z, h2, s[k]);
            s[k] = fmaf(w.w, h3, s[k]);
          }
        }
      }
      if (base + r < N) {
#pragma unroll
        for (int k = 0; k < K; k++) o[(size_t)(base + r) * NOUT + k0 + k] = s[k];
      }
    }
    __syncwarp();
  }
}

// Values of Ghat on its pattern from the head outputs,
//   Ghat_ii = softplus(dg_i + DIAG_OFFSET),  Ghat_ij = w_ij (a_i + u_i . v_j),
// with no constant term: a head near zero (the untrained network) gives
// Ghat = I, i.e. G G^T = D^-1, Jacobi; every off-diagonal value is learned.
// Optionally the scaled factor G = D^-1/2 Ghat for the apply, in G order and
// in G^T order.
__global__ void k_assemble(int nnzL, const int *__restrict__ grow,
                           const int *__restrict__ gcol,
                           const int *__restrict__ g2a,
                           const float *__restrict__ ahat,
                           const float *__restrict__ o, float *__restrict__ ghat,
                           const double *__restrict__ dis,
                           const int *__restrict__ g2t, float *__restrict__ gs,
                           float *__restrict__ gts, __nv_bfloat16 *__restrict__ sgv,
                           __nv_bfloat16 *__restrict__ stv,
                           const int *__restrict__ g2sg,
                           const int *__restrict__ t2st,
                           __nv_bfloat16 *__restrict__ gbv,
                           const int *__restrict__ g2b) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nnzL;
       e += gridDim.x * blockDim.x) {
    const int i = grow[e], j = gcol[e];
    // Rows of o are 8-byte aligned: pairs, all loaded before the first use.
    const float2 *oi = reinterpret_cast<const float2 *>(o + (size_t)i * NOUT);
    const float2 *oj = reinterpret_cast<const float2 *>(o + (size_t)j * NOUT + 2 + RANK);
    const float2 a = oi[0], u0 = oi[1], u1 = oi[2], v0 = oj[0], v1 = oj[1];
    const float w = fabsf(ahat[g2a[e]]);
    float v;
    if (i == j) {
      v = softplus(a.y + DIAG_OFFSET);
    } else {
      float uv = fmaf(u0.x, v0.x, 0.f);
      uv = fmaf(u0.y, v0.y, uv);
      uv = fmaf(u1.x, v1.x, uv);
      uv = fmaf(u1.y, v1.y, uv);
      v = w * (a.x + uv);
    }
    ghat[e] = v;
    if (gbv) {  // the band copy of G (BF16), which serves G and G^T
      gbv[g2b[e]] = __float2bfloat16_rn((float)(dis[i] * (double)v));
    } else if (sgv) {  // the SELL-U copies of G and G^T (BF16)
      const __nv_bfloat16 bv = __float2bfloat16_rn((float)(dis[i] * (double)v));
      sgv[g2sg[e]] = bv;
      stv[t2st[g2t[e]]] = bv;
    } else if (gs) {  // FP32 CRS copies when the SELL-U layouts do not fit
      const float sv = (float)(dis[i] * (double)v);
      gs[e] = sv;
      gts[g2t[e]] = sv;
    }
  }
}

// Rows of G (TRANS: of G^T, over G's entries t2g) for the sorted slices, with the
// values that k_assemble gives the other BF16 copies.
template <bool TRANS>
struct RowsFactor {
  const int *ptr, *idx, *t2g;
  const float *ghat;
  const double *dis;
  __device__ int begin(int i) const { return ptr[i]; }
  __device__ int end(int i) const { return ptr[i + 1]; }
  __device__ int col(int, int j) const { return idx[j]; }
  __device__ float val(int i, int j) const {
    return TRANS ? (float)(dis[idx[j]] * (double)ghat[t2g[j]])
                 : (float)(dis[i] * (double)ghat[j]);
  }
};

// ---------------------------------------------------------------------------
// Training: Adam, probes (the loss and its gradient: train.cuh)

// Adam (bias-corrected), in place.
__global__ void k_adam(int n, float *__restrict__ p, float *__restrict__ m,
                       float *__restrict__ v, const float *__restrict__ g,
                       float lr, float b1, float b2, float eps, int step) {
  const float c1 = 1.f - powf(b1, (float)step);
  const float c2 = 1.f - powf(b2, (float)step);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += gridDim.x * blockDim.x) {
    const float gk = g[k];
    const float mk = b1 * m[k] + (1.f - b1) * gk;
    const float vk = b2 * v[k] + (1.f - b2) * gk * gk;
    m[k] = mk;
    v[k] = vk;
    p[k] -= lr * (mk / c1) / (sqrtf(vk / c2) + eps);
  }
}

// Residual snapshot of the solver: s = sum_i (dis_i r_i)^2 over the FP64
// residual r = b - A x; the last CTA stores the unit-RMS scale sqrt(N / s).
__global__ void __launch_bounds__(kThreads)
    k_snap_norm(int N, const double *__restrict__ r,
                const double *__restrict__ dis, double *partials,
                unsigned *ticket, double *scale) {
  double a = 0.0;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < N;
       i += gridDim.x * kThreads) {
    const double v = dis[i] * r[i];
    a = fma(v, v, a);
  }
  double in[1] = {a}, out[1];
  if (grid_reduce<1>(in, partials, ticket, out) && threadIdx.x == 0)
    *scale = out[0] > 0.0 ? sqrt((double)N / out[0]) : 0.0;
}

// snap[i*S + col] = dis_i r_i * scale: the Jacobi-scaled residual with unit
// RMS, the coordinates of the scaled system the probes live in.
__global__ void k_snap_store(int N, const double *__restrict__ r,
                             const double *__restrict__ dis,
                             const double *__restrict__ scale,
                             float *__restrict__ snap, int col) {
  const double sc = *scale;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += gridDim.x * blockDim.x)
    snap[(size_t)i * S + col] = (float)(dis[i] * r[i] * sc);
}

// V[:, c0:S) = snap[:, c0:S) (the residual probe columns).
__global__ void k_copy_probe_cols(int N, const float *__restrict__ snap,
                                  float *__restrict__ V, int c0) {
  const size_t n = (size_t)N * S;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    if ((int)(i % S) >= c0) V[i] = snap[i];
}

// Rademacher probes from a counter-based hash: V[i*S+s] = +-1.
__global__ void k_rademacher(int N, unsigned long long seed, float *V) {
  const int total = N * S;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += gridDim.x * blockDim.x) {
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(t + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    V[t] = (z & 1ull) ? 1.f : -1.f;
  }
}

}  // namespace learned
}  // namespace cgx

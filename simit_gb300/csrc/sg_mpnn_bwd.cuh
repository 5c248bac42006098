// Backward kernels of the message-passing network (FP32, training meshes).
//
// Per vertex the backward pass is three small dense products (64x64, 64x8,
// 8x64) and one gather; per network the weight gradients are nine outer
// products summed over the vertices.  Both are tiled: a CTA stages a slab of
// vertices in shared memory and every thread keeps a 4x4 register tile, so a
// staged value is used 16 times instead of once.
#pragma once
#include "sg_mpnn.cuh"

namespace sg {
namespace mpnn {

constexpr int BW_V = 64;    // vertices per tile
constexpr int BW_T = 256;   // threads: 16 x 16, each 4 vertices x 4 columns
constexpr int BW_LD = 68;   // row stride of the 64-wide shared tiles (float4-aligned)

struct BwdSmem {
  float w[H * BW_LD];       // bf16-rounded 64x64 weights, [h][c]
  float dg[H * BW_LD];      // the tile's dg, transposed: [h][vertex]
  float m[H * K];           // message weights [h][j]
  float p[K * H];           // projection weights [j][h]
  float dq[BW_V * K];       // the tile's gathered cotangents [vertex][j]
};

// dm = Wm^T dg and dha = bf(Wh)^T dg of the tile (dg staged in S.dg).
__device__ __forceinline__ void bwd_products(BwdSmem &S, int64_t v0, int nv,
                                             float *__restrict__ dm, float *__restrict__ dha) {
#pragma unroll
  for (int e = 0; e < BW_V * K / BW_T; ++e) {
    const int t = threadIdx.x + e * BW_T, j = t % K, v = t / K;
    // four partial sums: a shorter rounding chain than one 64-term sum
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int h = 0; h < H; h += 4)
#pragma unroll
      for (int q = 0; q < 4; ++q) s[q] += S.m[(h + q) * K + j] * S.dg[(h + q) * BW_LD + v];
    if (v < nv) dm[(v0 + v) * K + j] = (s[0] + s[1]) + (s[2] + s[3]);
  }
  const int vt = (threadIdx.x >> 4) * 4, ct = (threadIdx.x & 15) * 4;
  float acc[4][4] = {};
#pragma unroll 8
  for (int h = 0; h < H; ++h) {
    const float4 d = *reinterpret_cast<const float4 *>(&S.dg[h * BW_LD + vt]);
    const float4 w = *reinterpret_cast<const float4 *>(&S.w[h * BW_LD + ct]);
    const float dv[4] = {d.x, d.y, d.z, d.w}, wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] += wv[j] * dv[i];
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (vt + i < nv)
      *reinterpret_cast<float4 *>(&dha[(v0 + vt + i) * H + ct]) =
          make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
}

// Weights of one layer into shared memory (Wh rounded to bf16 as the forward
// tensor-core operand is).
__device__ __forceinline__ void bwd_load_weights(BwdSmem &S, const float *__restrict__ prm,
                                                 int oWh, int oWm) {
  for (int e = threadIdx.x; e < H * H; e += BW_T)
    S.w[(e / H) * BW_LD + e % H] = bf16r(prm[oWh + e]);
  for (int e = threadIdx.x; e < H * K; e += BW_T) S.m[e] = prm[oWm + e];
}

// B1: dg3 = (Wout^T dz) * [g3 > 0]; dm3 = W3m^T dg3; dh2a = bf(W3h)^T dg3.
//
// Bound by its reads and writes of three 64-wide rows a vertex once the
// product is tiled.  One warp per vertex, reading each weight from L1 for
// one multiply-add, took 78 us at 35,937 vertices.
__global__ void __launch_bounds__(BW_T) k_b1(int32_t n, int lin, const float *__restrict__ prm,
                                             const float *__restrict__ dz,
                                             const float *__restrict__ g3,
                                             float *__restrict__ dg3, float *__restrict__ dm3,
                                             float *__restrict__ dh2a) {
  __shared__ __align__(16) BwdSmem S;
  bwd_load_weights(S, prm, O_W3H, O_W3M);
  const int h = threadIdx.x & (H - 1);
  const float w0 = prm[O_WOUT + h], w1 = prm[O_WOUT + H + h], w2 = prm[O_WOUT + 2 * H + h];
  for (int64_t v0 = (int64_t)blockIdx.x * BW_V; v0 < n; v0 += (int64_t)gridDim.x * BW_V) {
    const int nv = (int)min((int64_t)BW_V, n - v0);
    __syncthreads();
    for (int v = threadIdx.x / H; v < BW_V; v += BW_T / H) {
      float d = 0.f;
      if (v < nv) {
        const float *z = dz + (v0 + v) * 3;
        d = w0 * z[0] + w1 * z[1] + w2 * z[2];
        if (!lin && !(g3[(v0 + v) * H + h] > 0.f)) d = 0.f;
        dg3[(v0 + v) * H + h] = d;
      }
      S.dg[h * BW_LD + v] = d;
    }
    __syncthreads();
    bwd_products(S, v0, nv, dm3, dh2a);
  }
}

// Middle step: dq = sum_u a dm_u (K); dh = dha + P^T dq; dg = dh * [g > 0];
// optional dm_next = Wm^T dg (K), dha_next = bf(Wh)^T dg (H).  Bound by the
// gather's chain of dependent loads (one (vertex, message) pair a thread).
// The warp-per-vertex form took 59 us at 35,937 vertices.
__global__ void __launch_bounds__(BW_T) k_bmid(int32_t n, int lin,
                                               const uint32_t *__restrict__ rowptr,
                                               const uint32_t *__restrict__ colidx,
                                               const float *__restrict__ a,
                                               const float *__restrict__ prm, int oP, int oWm,
                                               int oWh, const float *__restrict__ dm,
                                               const float *__restrict__ dha,
                                               const float *__restrict__ g,
                                               float *__restrict__ dq, float *__restrict__ dgout,
                                               float *__restrict__ dm_next,
                                               float *__restrict__ dha_next) {
  __shared__ __align__(16) BwdSmem S;
  if (dm_next) bwd_load_weights(S, prm, oWh, oWm);
  for (int e = threadIdx.x; e < K * H; e += BW_T) S.p[e] = prm[oP + e];
  const int h = threadIdx.x & (H - 1);
  for (int64_t v0 = (int64_t)blockIdx.x * BW_V; v0 < n; v0 += (int64_t)gridDim.x * BW_V) {
    const int nv = (int)min((int64_t)BW_V, n - v0);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < BW_V * K / BW_T; ++e) {
      const int t = threadIdx.x + e * BW_T, j = t % K, v = t / K;
      float s = 0.f;
      if (v < nv) {
        const uint32_t q1 = rowptr[v0 + v + 1];
#pragma unroll 4
        for (uint32_t q = rowptr[v0 + v]; q < q1; ++q) s += a[q] * dm[(size_t)colidx[q] * K + j];
        dq[(v0 + v) * K + j] = s;
      }
      S.dq[t] = s;
    }
    __syncthreads();
    for (int v = threadIdx.x / H; v < BW_V; v += BW_T / H) {
      float d = 0.f;
      if (v < nv) {
        d = dha[(v0 + v) * H + h];
#pragma unroll
        for (int j = 0; j < K; ++j) d += S.p[j * H + h] * S.dq[v * K + j];
        if (!lin && !(g[(v0 + v) * H + h] > 0.f)) d = 0.f;
        dgout[(v0 + v) * H + h] = d;
      }
      S.dg[h * BW_LD + v] = d;
    }
    if (!dm_next) continue;
    __syncthreads();
    bwd_products(S, v0, nv, dm_next, dha_next);
  }
}

// Weight gradients of one network pass, all nine outer products in one
// launch: part[chunk][NPARAM] in the parameters' own layout, summed in chunk
// order by k_wgrad_sum.  Group y = 0: dW3h, dW3m, dP3; 1: dW2h, dW2m, dP2;
// 2: dW1s, dW1m, dWout.  A CTA stages WG_V vertices of both sides and each
// thread keeps a 4x4 tile of the 64x64 product and four entries of the
// 64x8 and 8x64 ones: 20 multiply-adds for six shared-memory loads, bound by
// issue.  At 35,937 vertices one pass takes about 20 us; one thread per
// product entry with both factors read from global memory took 4.1 ms.
// RELU / BF: the activation, and its bf16 rounding as the tensor-core
// operand (not with split activations).
constexpr int WG_V = 32;
constexpr int WG_C = H + K;
struct WgradArgs {
  int32_t n;
  int64_t rows;  // vertices per chunk
  const float *dz, *dg1, *dg2, *dg3, *dq2, *dq3;
  const float *g1, *g2, *g3, *s, *m1, *m2, *m3;
  float *part;
};
template <bool RELU> __device__ __forceinline__ float wg_act(float y) {
  return RELU ? fmaxf(y, 0.f) : y;
}
template <bool RELU, bool BF>
__global__ void __launch_bounds__(256) k_wgrad(WgradArgs a) {
  __shared__ __align__(16) float X[WG_V * WG_C], Y[WG_V * WG_C];
  const int grp = blockIdx.y, t = threadIdx.x;
  const int64_t v0 = (int64_t)blockIdx.x * a.rows, v1 = min((int64_t)a.n, v0 + a.rows);
  const float *gx = grp == 0 ? a.dg3 : grp == 1 ? a.dg2 : a.dg1;
  const float *gy = grp == 0 ? a.g2 : grp == 1 ? a.g1 : a.g3;
  const float *ex = grp == 0 ? a.dq3 : a.dq2, *ey = grp == 0 ? a.m3 : a.m2;
  const int ot = (t >> 4) * 4, it = (t & 15) * 4;
  float acc[4][4] = {}, am[2] = {}, ap[2] = {}, a1[3] = {};
  for (int64_t s0 = v0; s0 < v1; s0 += WG_V) {
    const int nv = (int)min((int64_t)WG_V, v1 - s0);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < WG_V * H / 4 / 256; ++e) {
      const int f = t + e * 256, v = f / (H / 4), c = (f % (H / 4)) * 4;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4 *>(&X[v * WG_C + c]) =
          v < nv ? *reinterpret_cast<const float4 *>(&gx[(s0 + v) * H + c]) : zero;
      *reinterpret_cast<float4 *>(&Y[v * WG_C + c]) =
          v < nv ? *reinterpret_cast<const float4 *>(&gy[(s0 + v) * H + c]) : zero;
    }
    {
      const int v = t / K, c = t % K;  // 256 = WG_V * K
      float xv = 0.f, yv = 0.f;
      if (v < nv) {
        if (grp < 2) {
          xv = ex[(s0 + v) * K + c];
          yv = ey[(s0 + v) * K + c];
        } else {
          if (c < 3) {
            xv = a.dz[(s0 + v) * 3 + c];
            yv = a.s[(s0 + v) * 3 + c];
          } else if (c < 6) {
            yv = a.m1[(s0 + v) * 3 + c - 3];
          }
        }
      }
      X[v * WG_C + H + c] = xv;
      Y[v * WG_C + H + c] = yv;
    }
    __syncthreads();
    if (grp < 2) {
#pragma unroll 2
      for (int v = 0; v < nv; ++v) {
        const float *xr = X + v * WG_C, *yr = Y + v * WG_C;
        const float4 x4 = *reinterpret_cast<const float4 *>(xr + ot);
        const float4 y4 = *reinterpret_cast<const float4 *>(yr + it);
        const float xv[4] = {x4.x, x4.y, x4.z, x4.w};
        float yv[4] = {y4.x, y4.y, y4.z, y4.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          yv[q] = wg_act<RELU>(yv[q]);
          if (BF) yv[q] = bf16r(yv[q]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] += xv[i] * yv[j];
        const float xm = xr[t >> 2];
        const float2 ym = *reinterpret_cast<const float2 *>(yr + H + (t & 3) * 2);
        am[0] += xm * ym.x;
        am[1] += xm * ym.y;
        const float xp = xr[H + (t >> 5)];
        const float2 yp = *reinterpret_cast<const float2 *>(yr + (t & 31) * 2);
        ap[0] += xp * wg_act<RELU>(yp.x);
        ap[1] += xp * wg_act<RELU>(yp.y);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int e = t + k * 256;
        if (e >= 9 * H) break;
        // entries 0..191 dW1s, 192..383 dW1m, 384..575 dWout
        const int q = e % (3 * H), which = e / (3 * H);
        const int xi = which == 2 ? H + q / H : q / 3;
        const int yi = which == 2 ? q % H : H + which * 3 + q % 3;
        float sum = 0.f;
        for (int v = 0; v < nv; ++v) {
          float y = Y[v * WG_C + yi];
          if (which == 2) y = wg_act<RELU>(y);
          sum += X[v * WG_C + xi] * y;
        }
        a1[k] += sum;
      }
    }
  }
  float *out = a.part + (size_t)blockIdx.x * NPARAM;
  if (grp < 2) {
    const int oh = grp == 0 ? O_W3H : O_W2H, om = grp == 0 ? O_W3M : O_W2M;
    const int op = grp == 0 ? O_P3 : O_P2;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<float4 *>(&out[oh + (ot + i) * H + it]) =
          make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    *reinterpret_cast<float2 *>(&out[om + (t >> 2) * K + (t & 3) * 2]) = make_float2(am[0], am[1]);
    *reinterpret_cast<float2 *>(&out[op + (t >> 5) * H + (t & 31) * 2]) =
        make_float2(ap[0], ap[1]);
  } else {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int e = t + k * 256;
      if (e >= 9 * H) break;
      const int q = e % (3 * H), which = e / (3 * H);
      out[(which == 0 ? O_W1S : which == 1 ? O_W1M : O_WOUT) + q] = a1[k];
    }
  }
}

// grad (= or +=) the chunks' sum: 32 parameters a CTA, its eight warps take
// an eighth of the chunks each, in a fixed order.
__global__ void __launch_bounds__(256) k_wgrad_sum(const float *__restrict__ part, int chunks,
                                                   int add, float *__restrict__ grad) {
  __shared__ float sh[8][32];
  const int e = blockIdx.x * 32 + (threadIdx.x & 31), w = threadIdx.x >> 5;
  const int c1 = (int)((int64_t)chunks * (w + 1) / 8);
  float s = 0.f;
  if (e < NPARAM)
#pragma unroll 8
    for (int c = (int)((int64_t)chunks * w / 8); c < c1; ++c) s += part[(size_t)c * NPARAM + e];
  sh[w][threadIdx.x & 31] = s;
  __syncthreads();
  if (w == 0 && e < NPARAM) {
    float tot = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) tot += sh[k][threadIdx.x];
    grad[e] = add ? grad[e] + tot : tot;
  }
}

}  // namespace mpnn
}  // namespace sg

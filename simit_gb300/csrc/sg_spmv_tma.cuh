// TMA-staged 3x3 blocked SpMV.
//
// A CTA walks tiles of ROWS consecutive block rows (persistent grid).  A
// tile's values and column indices are contiguous in the CSR arrays, so one
// thread issues two 1-D bulk copies (cp.async.bulk, 16-byte aligned head,
// the unaligned tail of at most 15 bytes loaded by threads) into one of two
// shared-memory buffers while the CTA computes the previous tile from the
// other.  HBM therefore sees full-line streaming reads of the matrix, and the
// compute side reads each block's 9 values from shared memory (lane stride 9
// words: bank-conflict free).  x is gathered through L1/L2; y is written by
// the group's lanes.  With DOT the kernel also returns the CTA's partial of
// p.q (the CG K1 epilogue).
#pragma once
#include "sg_solver_kernels.cuh"
#include "sg_tma.cuh"

#include <type_traits>

namespace sg {

template <typename MT, int BB = 9>
__host__ __device__ inline size_t tma_vbytes(int capb) {
  return (((size_t)capb * BB * sizeof(MT) + 32) + 15) & ~size_t(15);
}
__host__ __device__ inline size_t tma_cbytes(int capb) {
  return (((size_t)capb * 4 + 32) + 15) & ~size_t(15);
}
template <typename MT> inline size_t tma_smem_bytes(int capb, int nst) {
  const size_t b = 64 + (size_t)nst * (tma_vbytes<MT>(capb) + tma_cbytes(capb));
  return b > SUM_SMEM ? b : SUM_SMEM;
}

// y_r = (A x)_r for block row r (blocks [rb, e)) from its tile's values vb and
// columns cb (block q at vb[q*9 - voff], cb[q - coff]); G lanes per row, lane
// gl takes blocks rb + gl, + G, ...  The first U blocks of each lane (rows of up
// to 24 blocks) use a fixed, predicated trip count so all of the lane's x
// gathers are in flight at once; the remainder loop keeps the same
// accumulation order.  With DOT, acc accumulates x_r . y_r (DotAcc).
template <int G, typename MT, typename VT, bool DOT>
__device__ __forceinline__ void tile_row(int64_t r, int gl, unsigned mask,
                                         uint32_t rb, uint32_t e,
                                         const MT *__restrict__ vb,
                                         const uint32_t *__restrict__ cb, size_t voff,
                                         size_t coff, const VT *__restrict__ x,
                                         VT *__restrict__ y, DotAcc<VT> &acc) {
  VT a0 = 0, a1 = 0, a2 = 0;
  constexpr int U = (24 + G - 1) / G;
  const uint32_t q0 = rb + gl;
  VT xg[U][3], xr = 0;
  if (DOT && G >= 3 && gl < 3) xr = x[(size_t)r * 3 + gl];  // in flight with the gathers
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const uint32_t q = q0 + k * G;
    if (q < e) {
      const uint32_t c = cb[q - coff];
      xg[k][0] = ldg(x + (size_t)c * 3 + 0);
      xg[k][1] = ldg(x + (size_t)c * 3 + 1);
      xg[k][2] = ldg(x + (size_t)c * 3 + 2);
    }
  }
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const uint32_t q = q0 + k * G;
    if (q < e) {
      const MT *v = vb + ((size_t)q * 9 - voff);
      const VT x0 = xg[k][0], x1 = xg[k][1], x2 = xg[k][2];
      a0 += (VT)v[0] * x0 + (VT)v[1] * x1 + (VT)v[2] * x2;
      a1 += (VT)v[3] * x0 + (VT)v[4] * x1 + (VT)v[5] * x2;
      a2 += (VT)v[6] * x0 + (VT)v[7] * x1 + (VT)v[8] * x2;
    }
  }
#pragma unroll 4
  for (uint32_t q = q0 + U * G; q < e; q += G) {
    const uint32_t c = cb[q - coff];
    const MT *v = vb + ((size_t)q * 9 - voff);
    const VT x0 = ldg(x + (size_t)c * 3 + 0), x1 = ldg(x + (size_t)c * 3 + 1),
             x2 = ldg(x + (size_t)c * 3 + 2);
    a0 += (VT)v[0] * x0 + (VT)v[1] * x1 + (VT)v[2] * x2;
    a1 += (VT)v[3] * x0 + (VT)v[4] * x1 + (VT)v[5] * x2;
    a2 += (VT)v[6] * x0 + (VT)v[7] * x1 + (VT)v[8] * x2;
  }
  a0 = group_sum<G>(a0, mask);
  a1 = group_sum<G>(a1, mask);
  a2 = group_sum<G>(a2, mask);
  if (G >= 3) {
    if (gl < 3) {
      const VT yv = gl == 0 ? a0 : (gl == 1 ? a1 : a2);
      y[(size_t)r * 3 + gl] = yv;
      if (DOT) acc.add(xr, yv);
    }
  } else if (gl == 0) {  // fewer than 3 lanes: lane 0 writes the row
    y[(size_t)r * 3 + 0] = a0;
    y[(size_t)r * 3 + 1] = a1;
    y[(size_t)r * 3 + 2] = a2;
    if (DOT) {
      acc.add(x[(size_t)r * 3], a0);
      acc.add(x[(size_t)r * 3 + 1], a1);
      acc.add(x[(size_t)r * 3 + 2], a2);
    }
  }
}

// Scalar CSR row (1x1 blocks): y_r = sum_q vb[q - voff] x[cb[q - coff]],
// same lane split, predicated gathers and accumulation order as tile_row.
template <int G, typename MT, typename VT, bool DOT>
__device__ __forceinline__ void tile_row1(int64_t r, int gl, unsigned mask,
                                          uint32_t rb, uint32_t e,
                                          const MT *__restrict__ vb,
                                          const uint32_t *__restrict__ cb, size_t voff,
                                          size_t coff, const VT *__restrict__ x,
                                          VT *__restrict__ y, DotAcc<VT> &acc) {
  VT a = 0;
  constexpr int U = (24 + G - 1) / G;
  const uint32_t q0 = rb + gl;
  VT xg[U], xr = 0;
  if (DOT && gl == 0) xr = x[r];
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const uint32_t q = q0 + k * G;
    if (q < e) xg[k] = ldg(x + cb[q - coff]);
  }
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const uint32_t q = q0 + k * G;
    if (q < e) a += (VT)vb[q - voff] * xg[k];
  }
#pragma unroll 4
  for (uint32_t q = q0 + U * G; q < e; q += G) a += (VT)vb[q - voff] * ldg(x + cb[q - coff]);
  a = group_sum<G>(a, mask);
  if (gl == 0) {
    y[r] = a;
    if (DOT) acc.add(xr, a);
  }
}

// NST-stage pipeline: while the CTA computes tile k, the copies of tiles
// k+1 .. k+NST-1 are in flight.  A tile of more than capb blocks (the
// buffers' capacity) is never staged: it is read straight from global
// memory, so a stale tile statistic costs speed, never memory safety.
template <int G, int ROWS, int NST, typename MT, typename VT, bool DOT>
__global__ void __launch_bounds__(ROWS *G)
    k_bsr3_tma(const SolveCtl *__restrict__ ctl, int32_t n, const uint32_t *__restrict__ rowptr,
               const uint32_t *__restrict__ colidx, const MT *__restrict__ vals,
               const VT *__restrict__ x, VT *__restrict__ y, double *__restrict__ part, int capb,
               int *err) {
  static_assert(NST >= 2 && NST <= 6, "stages");
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int ok_flag;
  if (ctl && ctl->status != ST_RUNNING) return;
  const size_t vbytes = tma_vbytes<MT>(capb), cbytes = tma_cbytes(capb);
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm);
  unsigned char *base = sm + 64;
  auto vbuf = [&](int b) { return reinterpret_cast<MT *>(base + (size_t)b * (vbytes + cbytes)); };
  auto cbuf = [&](int b) {
    return reinterpret_cast<uint32_t *>(base + (size_t)b * (vbytes + cbytes) + vbytes);
  };
  const int ntiles = (n + ROWS - 1) / ROWS;
  constexpr size_t S = sizeof(MT);
  if (threadIdx.x == 0) {
    for (int b = 0; b < NST; ++b) mbar_init(&bar[b], 1);
    mbar_fence_init();
  }
  __syncthreads();

  auto tile_range = [&](int tile, uint32_t &b0, uint32_t &b1) {
    const int r0 = tile * ROWS;
    const int r1 = min(n, r0 + ROWS);
    b0 = rowptr[r0];
    b1 = rowptr[r1];
  };
  auto issue = [&](int tile, int b) {
    uint32_t b0, b1;
    tile_range(tile, b0, b1);
    const size_t vs = ((size_t)b0 * 9 * S) & ~size_t(15), ve = ((size_t)b1 * 9 * S) & ~size_t(15);
    const size_t cs = ((size_t)b0 * 4) & ~size_t(15), ce = ((size_t)b1 * 4) & ~size_t(15);
    fence_proxy_async_smem();
    if (b1 - b0 > (uint32_t)capb) {  // larger than the buffers: read from global
      mbar_arrive_expect_tx(&bar[b], 0);
      return;
    }
    mbar_arrive_expect_tx(&bar[b], (uint32_t)((ve - vs) + (ce - cs)));
    if (ve > vs)
      bulk_g2s(vbuf(b), reinterpret_cast<const unsigned char *>(vals) + vs, (uint32_t)(ve - vs),
               &bar[b]);
    if (ce > cs)
      bulk_g2s(cbuf(b), reinterpret_cast<const unsigned char *>(colidx) + cs,
               (uint32_t)(ce - cs), &bar[b]);
  };

  const int gl = threadIdx.x & (G - 1);
  const unsigned mask = group_mask<G>();
  DotAcc<VT> acc;
  // local tile k of this CTA is global tile blockIdx.x + k*gridDim.x
  const int my_tiles = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  if (threadIdx.x == 0)
    for (int k = 0; k < NST - 1 && k < my_tiles; ++k) issue(blockIdx.x + k * gridDim.x, k);
  for (int k = 0; k < my_tiles; ++k) {
    const int b = k % NST;
    const int tile = blockIdx.x + k * gridDim.x;
    if (threadIdx.x == 0) {
      const int kn = k + NST - 1;
      if (kn < my_tiles) issue(blockIdx.x + kn * gridDim.x, kn % NST);
      const bool ok = mbar_wait(&bar[b], (uint32_t)((k / NST) & 1));
      ok_flag = ok ? 1 : 0;
      if (!ok) {
        atomicCAS(err, 0, 6 /* DEV_TMA_TIMEOUT */);
        // no new copies; wait (bounded) on every barrier with a copy still
        // in flight, this tile's included, before leaving; if one of those
        // waits runs out too, a copy may still land in shared memory after
        // the CTA exits: record that (the results are then undefined and
        // the context should be reset)
        bool drained = true;
        for (int kk = k; kk < my_tiles && kk <= kn; ++kk)
          drained = mbar_wait(&bar[kk % NST], (uint32_t)((kk / NST) & 1)) && drained;
        if (!drained) atomicExch(err, 8 /* DEV_TMA_UNDRAINED */);
      }
    }
    __syncthreads();
    if (!ok_flag) break;
    uint32_t b0, b1;
    tile_range(tile, b0, b1);
    const bool staged = b1 - b0 <= (uint32_t)capb;
    const size_t vs = staged ? ((size_t)b0 * 9 * S) & ~size_t(15) : 0;
    const size_t cs = staged ? ((size_t)b0 * 4) & ~size_t(15) : 0;
    if (staged) {
      // unaligned tails (< 16 bytes each)
      const size_t ve = ((size_t)b1 * 9 * S) & ~size_t(15), ce = ((size_t)b1 * 4) & ~size_t(15);
      const int vt = (int)(((size_t)b1 * 9 * S - ve) / S);
      const int ct = (int)(((size_t)b1 * 4 - ce) / 4);
      if ((int)threadIdx.x < vt) vbuf(b)[(ve - vs) / S + threadIdx.x] = vals[ve / S + threadIdx.x];
      if ((int)threadIdx.x >= 32 && (int)threadIdx.x < 32 + ct)
        cbuf(b)[(ce - cs) / 4 + threadIdx.x - 32] = colidx[ce / 4 + threadIdx.x - 32];
    }
    __syncthreads();
    const int r = tile * ROWS + (int)(threadIdx.x / G);
    if (r < n) {
      // two inlined copies: shared-memory loads for a staged tile, global
      // loads for an oversize one
      if (staged)
        tile_row<G, MT, VT, DOT>(r, gl, mask, rowptr[r], rowptr[r + 1], vbuf(b), cbuf(b), vs / S,
                                 cs / 4, x, y, acc);
      else
        tile_row<G, MT, VT, DOT>(r, gl, mask, rowptr[r], rowptr[r + 1], vals, colidx, 0, 0, x, y,
                                 acc);
    }
    __syncthreads();
  }
  if (DOT) {  // CG K1: the last CTA leaves the p.q total in ctl->pq_tot
    const double v = acc.value();
    double t, tot;
    block_sums<1>(&v, &t, sum_buf(sm));
    SolveCtl *c = const_cast<SolveCtl *>(ctl);
    if (finalize_partials<1>(&t, part, &c->tick1, &tot, sum_buf(sm)) && threadIdx.x == 0)
      c->pq_tot = tot;
  }
}

}  // namespace sg

namespace sg {

// Per-warp variant: every warp runs its own NST-stage bulk-copy pipeline
// over tiles of RW = 32/G consecutive block rows (global warp w takes tiles
// w, w + total warps, ...), waits on its own mbarriers and synchronises only
// with __syncwarp, so no warp waits for another's copy or compute.  Each
// warp's buffers hold capb blocks; a larger tile (the caller's statistics
// were stale, or a very long row) is read straight from global memory.
constexpr int WTMA_WARPS = 4;

template <typename MT, int BB = 9> inline size_t wtma_smem_bytes(int capb, int nst) {
  const size_t b = (((size_t)WTMA_WARPS * nst * 8 + 15) & ~size_t(15)) +
                   (size_t)WTMA_WARPS * nst * (tma_vbytes<MT, BB>(capb) + tma_cbytes(capb));
  return b > SUM_SMEM ? b : SUM_SMEM;
}

// Body shared by the 3x3 (BS = 3) and scalar CSR (BS = 1) kernels.  A warp
// tile is P passes of 32/G rows (P > 1 makes the bulk copies of short
// scalar rows larger).
template <int BS, int G, int NST, int P, typename MT, typename VT, bool DOT>
__device__ __forceinline__ void wtma_body(const SolveCtl *__restrict__ ctl, int32_t n,
                                          const uint32_t *__restrict__ rowptr,
                                          const uint32_t *__restrict__ colidx,
                                          const MT *__restrict__ vals, const VT *__restrict__ x,
                                          VT *__restrict__ y, double *__restrict__ part,
                                          int capb, int *err, unsigned char *sm) {
  static_assert(NST >= 2 && NST <= 6, "stages");
  static_assert(BS == 1 || BS == 3, "block size");
  constexpr int RW = 32 / G * P;
  constexpr int BB = BS * BS;
  constexpr size_t S = sizeof(MT);
  pdl_wait_and_release();
  if (ctl && ctl->status != ST_RUNNING) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t vbytes = tma_vbytes<MT, BB>(capb), cbytes = tma_cbytes(capb);
  const size_t stage = vbytes + cbytes;
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm) + warp * NST;
  unsigned char *base =
      sm + (((size_t)WTMA_WARPS * NST * 8 + 15) & ~size_t(15)) + (size_t)warp * NST * stage;
  auto vbuf = [&](int b) { return reinterpret_cast<MT *>(base + (size_t)b * stage); };
  auto cbuf = [&](int b) { return reinterpret_cast<uint32_t *>(base + (size_t)b * stage + vbytes); };
  if (lane == 0) {
    for (int b = 0; b < NST; ++b) mbar_init(&bar[b], 1);
    mbar_fence_init();
  }
  __syncwarp();
  const int64_t ntiles = ((int64_t)n + RW - 1) / RW;
  const int64_t gw = (int64_t)blockIdx.x * WTMA_WARPS + warp;
  const int64_t nw = (int64_t)gridDim.x * WTMA_WARPS;
  const int64_t my = gw < ntiles ? (ntiles - 1 - gw) / nw + 1 : 0;
  // Row pointers of tiles k .. k + NST, a lane each (value i of a tile in
  // lane i % 32 of register i / 32), fetched a tile before they are needed:
  // neither the copies nor the rows wait for them.
  constexpr int NRP = RW / 32 + 1;
  uint32_t rp[NST + 1][NRP];
  auto fetch = [&](int64_t k, uint32_t *o) {
    const int64_t r0 = (gw + k * nw) * RW;
#pragma unroll
    for (int j = 0; j < NRP; ++j) {
      const int64_t i = min((int64_t)n, r0 + min(RW, 32 * j + lane));
      o[j] = k < my ? rowptr[i] : 0u;
    }
  };
  auto pointer = [&](const uint32_t *o, int i) {
    return __shfl_sync(0xffffffffu, o[i / 32], i % 32);
  };
  // A tile's copies are rounded up to 16 bytes where the matrix goes on
  // behind it; vlim, clim: the last 16-byte boundary inside the arrays.
  const size_t vlim = ((size_t)rowptr[n] * BB * S) & ~size_t(15);
  const size_t clim = ((size_t)rowptr[n] * 4) & ~size_t(15);
  auto up = [](size_t bytes, size_t lim) { return min((bytes + 15) & ~size_t(15), lim); };
  auto issue = [&](uint32_t b0, uint32_t b1, int b) {
    const size_t vs = ((size_t)b0 * BB * S) & ~size_t(15), ve = up((size_t)b1 * BB * S, vlim);
    const size_t cs = ((size_t)b0 * 4) & ~size_t(15), ce = up((size_t)b1 * 4, clim);
    fence_proxy_async_smem();
    if (b1 - b0 > (uint32_t)capb) {  // larger than the buffers: read from global
      mbar_arrive_expect_tx(&bar[b], 0);
      return;
    }
    const uint32_t vb = ve > vs ? (uint32_t)(ve - vs) : 0u, cb = ce > cs ? (uint32_t)(ce - cs) : 0u;
    mbar_arrive_expect_tx(&bar[b], vb + cb);
    if (vb) bulk_g2s(vbuf(b), reinterpret_cast<const unsigned char *>(vals) + vs, vb, &bar[b]);
    if (cb) bulk_g2s(cbuf(b), reinterpret_cast<const unsigned char *>(colidx) + cs, cb, &bar[b]);
  };
#pragma unroll
  for (int k = 0; k < NST; ++k) fetch(k, rp[k]);
#pragma unroll
  for (int k = 0; k < NST - 1; ++k) {
    const uint32_t b0 = pointer(rp[k], 0), b1 = pointer(rp[k], RW);
    if (lane == 0 && k < my) issue(b0, b1, k);
  }
  const int gl = lane & (G - 1);
  const unsigned mask = group_mask<G>();
  DotAcc<VT> acc;
  for (int64_t k = 0; k < my; ++k) {
    const int b = (int)(k % NST);
    const int64_t tile = gw + k * nw;
    const int64_t kn = k + NST - 1;
    {
      const uint32_t b0 = pointer(rp[NST - 1], 0), b1 = pointer(rp[NST - 1], RW);
      if (lane == 0 && kn < my) issue(b0, b1, (int)(kn % NST));
    }
    fetch(k + NST, rp[NST]);
    const bool ok = __all_sync(0xffffffffu, mbar_wait(&bar[b], (uint32_t)((k / NST) & 1)));
    if (!ok) {
      if (lane == 0) {
        atomicCAS(err, 0, 6 /* DEV_TMA_TIMEOUT */);
        // drain every barrier with a copy in flight (see k_bsr3_tma)
        bool drained = true;
        for (int64_t kk = k; kk < my && kk <= kn; ++kk)
          drained = mbar_wait(&bar[kk % NST], (uint32_t)((kk / NST) & 1)) && drained;
        if (!drained) atomicExch(err, 8 /* DEV_TMA_UNDRAINED */);
      }
      break;
    }
    const int64_t r0 = tile * RW;
    const uint32_t b0 = pointer(rp[0], 0), b1 = pointer(rp[0], RW);
    const bool staged = b1 - b0 <= (uint32_t)capb;
    const size_t vs = staged ? ((size_t)b0 * BB * S) & ~size_t(15) : 0;
    const size_t cs = staged ? ((size_t)b0 * 4) & ~size_t(15) : 0;
    if (staged && ((size_t)b1 * BB * S > vlim || (size_t)b1 * 4 > clim)) {
      // the matrix's end: unaligned tails (< 16 bytes each)
      const size_t ve = max(vs, up((size_t)b1 * BB * S, vlim)), ce = max(cs, up((size_t)b1 * 4, clim));
      if (ve / S + lane < (size_t)b1 * BB)
        vbuf(b)[(ve - vs) / S + lane] = vals[ve / S + lane];
      if (ce / 4 + lane < b1) cbuf(b)[(ce - cs) / 4 + lane] = colidx[ce / 4 + lane];
      __syncwarp();
    }
#pragma unroll
    for (int pp = 0; pp < P; ++pp) {
      const int i = pp * (32 / G) + lane / G;  // the row within the tile
      constexpr int NP = NRP - 1;
      const int j = pp * (32 / G) / 32;
      const uint32_t rb = __shfl_sync(0xffffffffu, rp[0][j], i % 32);
      uint32_t re = __shfl_sync(0xffffffffu, rp[0][j], (i + 1) % 32);
      if (NP > 0) {
        const uint32_t re2 = __shfl_sync(0xffffffffu, rp[0][min(j + 1, NP)], (i + 1) % 32);
        if ((i + 1) / 32 != j) re = re2;
      }
      const int64_t r = r0 + i;
      if (r < n) {
        if (BS == 3) {
          if (staged)
            tile_row<G, MT, VT, DOT>(r, gl, mask, rb, re, vbuf(b), cbuf(b), vs / S, cs / 4, x, y,
                                     acc);
          else
            tile_row<G, MT, VT, DOT>(r, gl, mask, rb, re, vals, colidx, 0, 0, x, y, acc);
        } else {
          if (staged)
            tile_row1<G, MT, VT, DOT>(r, gl, mask, rb, re, vbuf(b), cbuf(b), vs / S, cs / 4, x, y,
                                      acc);
          else
            tile_row1<G, MT, VT, DOT>(r, gl, mask, rb, re, vals, colidx, 0, 0, x, y, acc);
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < NST; ++t)
#pragma unroll
      for (int j = 0; j < NRP; ++j) rp[t][j] = rp[t + 1][j];
  }
  if (DOT) {  // CG K1: the last CTA leaves the p.q total in ctl->pq_tot
    const double v = acc.value();
    double t, tot;
    block_sums<1>(&v, &t, sum_buf(sm));
    SolveCtl *c = const_cast<SolveCtl *>(ctl);
    if (finalize_partials<1>(&t, part, &c->tick1, &tot, sum_buf(sm)) && threadIdx.x == 0)
      c->pq_tot = tot;
  }
}

template <int G, int NST, typename MT, typename VT, bool DOT>
__global__ void __launch_bounds__(WTMA_WARPS * 32)
    k_bsr3_wtma(const SolveCtl *__restrict__ ctl, int32_t n, const uint32_t *__restrict__ rowptr,
                const uint32_t *__restrict__ colidx, const MT *__restrict__ vals,
                const VT *__restrict__ x, VT *__restrict__ y, double *__restrict__ part,
                int capb, int *err) {
  extern __shared__ __align__(16) unsigned char sm[];
  wtma_body<3, G, NST, 1, MT, VT, DOT>(ctl, n, rowptr, colidx, vals, x, y, part, capb, err, sm);
}

// Scalar CSR (bs = 1) with the same per-warp pipeline, tiles of P passes.
template <int G, int NST, int P, typename MT, typename VT, bool DOT>
__global__ void __launch_bounds__(WTMA_WARPS * 32)
    k_csr_wtma(const SolveCtl *__restrict__ ctl, int32_t n, const uint32_t *__restrict__ rowptr,
               const uint32_t *__restrict__ colidx, const MT *__restrict__ vals,
               const VT *__restrict__ x, VT *__restrict__ y, double *__restrict__ part,
               int capb, int *err) {
  extern __shared__ __align__(16) unsigned char sm[];
  wtma_body<1, G, NST, P, MT, VT, DOT>(ctl, n, rowptr, colidx, vals, x, y, part, capb, err, sm);
}

// FP64 3x3 blocked SpMV, rows sorted by length inside a tile.
//
// An SM of this GPU has one FP64 pipe that takes a warp instruction every 16
// cycles, however many of the warp's lanes are active, so the product is bound
// by FP64 warp instructions (0.40 ms at 128^3: 9 multiply-adds a block in full
// warps) before it is by memory (0.33 ms).  Here a lane owns one component of
// one row: 3 multiply-adds a block, no reduction across lanes.  A CTA stages
// the values and columns of F64_ROWS rows with one bulk copy each, ranks the
// rows by length meanwhile, and gives each warp 32 (row, component) pairs of
// neighbouring rank, so that the lanes of a warp end together (the five-tet
// lattice alternates rows of 7 and 19 blocks).  With 4 lanes a row, two thirds
// of the multiply-adds' lanes and all of the shuffled additions were idle work.
// At 128^3: 0.555 ms, streaming with 4 lanes a row 1.04; 64^3: 85 us, 142.
// 64 rows: six full warps; three CTAs an SM keep the copies of two in flight
// (32 rows, six CTAs: 0.58 ms; 96 rows, two: 0.70).  Groups of 2, 6 or 8
// gathers instead of 4: 0.548 to 0.556; predicated groups: 0.60 (4), 0.77 (6).
// A row's two sums (even and odd blocks) round more often in sequence than the
// partial sums of 4 lanes: with random entries the rms error is 1.7e-16 of the
// result against 1.2e-16.  Four sums, 1.4e-16, take 0.572 ms; eight, 1.25e-16,
// 0.614: each further sum is an addition on the pipe that bounds the product.
constexpr int F64_ROWS = 64, F64_T = 3 * F64_ROWS;
constexpr int F64_U = 4;  // blocks whose gathers a lane has in flight
inline size_t f64_smem_bytes(int capb) {
  const size_t b = 16 + tma_vbytes<double>(capb) + tma_cbytes(capb);
  return b > SUM_SMEM ? b : SUM_SMEM;
}

template <bool DOT>
__device__ __forceinline__ void f64_task(uint32_t q0, uint32_t q1, int64_t row, int comp,
                                         const double *vb, const uint32_t *cb, size_t voff,
                                         size_t coff, const double *__restrict__ x,
                                         double *__restrict__ y, DotAcc<double> &acc) {
  double a[2] = {0.0, 0.0};  // even and odd blocks: half the dependent chain
  // U blocks, their gathers in flight together.  Whole groups only: a
  // predicated-off multiply-add still takes its place on the pipe.
  auto group = [&](auto width) {
    constexpr int U = decltype(width)::value;
    double xg[U][3];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const double *xc = x + (size_t)cb[q0 + k - coff] * 3;
      xg[k][0] = ldg(xc);
      xg[k][1] = ldg(xc + 1);
      xg[k][2] = ldg(xc + 2);
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const double *v = vb + ((size_t)(q0 + k) * 9 + comp * 3 - voff);
      a[k & 1] = fma(v[2], xg[k][2], fma(v[1], xg[k][1], fma(v[0], xg[k][0], a[k & 1])));
    }
    q0 += U;
  };
  while (q0 + F64_U <= q1) group(std::integral_constant<int, F64_U>());
  if (q0 + 2 <= q1) group(std::integral_constant<int, 2>());
  if (q0 < q1) group(std::integral_constant<int, 1>());
  const double yv = a[0] + a[1];
  y[row * 3 + comp] = yv;
  if (DOT) acc.add(x[row * 3 + comp], yv);
}

template <bool DOT>
__global__ void __launch_bounds__(F64_T, 3)
    k_bsr3_f64(const SolveCtl *__restrict__ ctl, int32_t n, const uint32_t *__restrict__ rowptr,
               const uint32_t *__restrict__ colidx, const double *__restrict__ vals,
               const double *__restrict__ x, double *__restrict__ y, double *__restrict__ part,
               int capb, int *err) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ uint32_t rp[F64_ROWS + 1];
  __shared__ uint8_t order[F64_ROWS];
  if (ctl && ctl->status != ST_RUNNING) return;
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm);
  double *vb = reinterpret_cast<double *>(sm + 16);
  uint32_t *cb = reinterpret_cast<uint32_t *>(sm + 16 + tma_vbytes<double>(capb));
  const int tid = threadIdx.x;
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
  }
  const int ntiles = (n + F64_ROWS - 1) / F64_ROWS;
  DotAcc<double> acc;
  uint32_t phase = 0, next = 0;  // next: the next tile's row pointers, a thread each
  if (tid <= F64_ROWS && (int)blockIdx.x < ntiles)
    next = rowptr[min((int64_t)n, (int64_t)blockIdx.x * F64_ROWS + tid)];
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t r0 = (int64_t)tile * F64_ROWS;
    const int nr = (int)min((int64_t)F64_ROWS, n - r0);
    __syncthreads();  // the previous tile's buffers and tables are free
    if (tid <= F64_ROWS) rp[tid] = next;
    __syncthreads();
    const uint32_t b0 = rp[0], b1 = rp[nr];
    const bool staged = b1 - b0 <= (uint32_t)capb;
    const size_t vs = staged ? ((size_t)b0 * 72) & ~size_t(15) : 0;
    const size_t cs = staged ? ((size_t)b0 * 4) & ~size_t(15) : 0;
    const size_t ve = ((size_t)b1 * 72) & ~size_t(15), ce = ((size_t)b1 * 4) & ~size_t(15);
    if (staged && tid == 0) {
      fence_proxy_async_smem();
      const uint32_t vn = ve > vs ? (uint32_t)(ve - vs) : 0u, cn = ce > cs ? (uint32_t)(ce - cs) : 0u;
      mbar_arrive_expect_tx(bar, vn + cn);
      if (vn) bulk_g2s(vb, reinterpret_cast<const unsigned char *>(vals) + vs, vn, bar);
      if (cn) bulk_g2s(cb, reinterpret_cast<const unsigned char *>(colidx) + cs, cn, bar);
    }
    // meanwhile: the rows by length, longest first, and the next row pointers
    if (tid < nr) {
      const uint32_t len = rp[tid + 1] - rp[tid];
      int rank = 0;
      for (int u = 0; u < nr; ++u) {
        const uint32_t lu = rp[u + 1] - rp[u];
        rank += lu > len || (lu == len && u < tid);
      }
      order[rank] = (uint8_t)tid;
    }
    if (tid <= F64_ROWS && tile + (int)gridDim.x < ntiles)
      next = rowptr[min((int64_t)n, r0 + (int64_t)gridDim.x * F64_ROWS + tid)];
    if (staged) {
      // the tails of less than 16 bytes
      if (tid >= 32 && tid < 32 + (int)((((size_t)b1 * 72) - ve) / 8))
        vb[(ve - vs) / 8 + tid - 32] = vals[ve / 8 + tid - 32];
      if (tid >= 64 && tid < 64 + (int)((((size_t)b1 * 4) - max(ce, cs)) / 4))
        cb[(max(ce, cs) - cs) / 4 + tid - 64] = colidx[max(ce, cs) / 4 + tid - 64];
      bool ok = mbar_wait(bar, phase);
      if (!ok) {
        if (tid == 0) {
          atomicCAS(err, 0, 6 /* DEV_TMA_TIMEOUT */);
          if (!mbar_wait(bar, phase)) atomicExch(err, 8 /* DEV_TMA_UNDRAINED */);
        }
      }
      if (__syncthreads_or(!ok)) break;
      phase ^= 1u;
    } else {
      __syncthreads();
    }
    const int rank = tid / 3, comp = tid - rank * 3;
    if (rank < nr) {
      const int rl = order[rank];
      if (staged)
        f64_task<DOT>(rp[rl], rp[rl + 1], r0 + rl, comp, vb, cb, vs / 8, cs / 4, x, y, acc);
      else
        f64_task<DOT>(rp[rl], rp[rl + 1], r0 + rl, comp, vals, colidx, 0, 0, x, y, acc);
    }
  }
  if (DOT) {  // CG K1: the last CTA leaves the p.q total in ctl->pq_tot
    const double v = acc.value();
    double t, tot;
    block_sums<1>(&v, &t, sum_buf(sm));
    SolveCtl *c = const_cast<SolveCtl *>(ctl);
    if (finalize_partials<1>(&t, part, &c->tick1, &tot, sum_buf(sm)) && threadIdx.x == 0)
      c->pq_tot = tot;
  }
}

// FP64 scalar row, one lane per row, called by the whole warp (a lane without
// a row passes rb = re).  Entries go 8 at a time, their gathers in flight together,
// the rest in one group of the exact width (a predicated-off multiply-add
// still takes its place on the pipe); lanes whose row has ended add 0 * 0.
// Even and odd entries have a sum each: half the dependent chain, and the
// additions of two lanes per row (rms error 1.11e-16 of the result either way).
template <bool DOT>
__device__ __forceinline__ void csr_row_f64(int64_t r, bool row, uint32_t rb, uint32_t re,
                                            const double *__restrict__ vb,
                                            const uint32_t *__restrict__ cb, size_t voff,
                                            size_t coff, const double *__restrict__ x,
                                            double *__restrict__ y, DotAcc<double> &acc) {
  const uint32_t longest = __reduce_max_sync(0xffffffffu, re - rb);
  double a[2] = {0.0, 0.0}, xr = 0.0;
  if (DOT && row) xr = x[r];
  uint32_t k = 0;
  auto group = [&](auto width) {
    constexpr int U = decltype(width)::value;
    double xg[U], vg[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const uint32_t q = rb + k + j;
      xg[j] = vg[j] = 0.0;
      if (q < re) {
        xg[j] = ldg(x + cb[q - coff]);
        vg[j] = vb[q - voff];
      }
    }
#pragma unroll
    for (int j = 0; j < U; ++j) a[j & 1] = fma(vg[j], xg[j], a[j & 1]);
    k += U;
  };
  while (k + 8 <= longest) group(std::integral_constant<int, 8>());
  switch (longest - k) {
    case 7: group(std::integral_constant<int, 7>()); break;
    case 6: group(std::integral_constant<int, 6>()); break;
    case 5: group(std::integral_constant<int, 5>()); break;
    case 4: group(std::integral_constant<int, 4>()); break;
    case 3: group(std::integral_constant<int, 3>()); break;
    case 2: group(std::integral_constant<int, 2>()); break;
    case 1: group(std::integral_constant<int, 1>()); break;
    default: break;
  }
  const double yv = a[0] + a[1];
  if (row) {
    y[r] = yv;
    if (DOT) acc.add(xr, yv);
  }
}

// FP64 scalar SpMV, a lane per row, rows sorted by length inside a warp's
// tile.  Bound by the FP64 pipe, which takes a warp's multiply-add every 16
// cycles whether 32 lanes use it or one.  G lanes per row waste lanes where G
// does not divide the row and add shuffle sums on the same pipe; a lane per
// row wastes what its row is shorter than the warp's longest.  So a warp
// takes C1_ROWS rows at a time, copies their values and columns to shared
// memory (one bulk copy each), sorts the rows by length meanwhile (radix sort
// on the bits in which the lengths differ, by ballots: no order depends on
// timing), and takes them in two passes of like rows: the 64^3 heat lattice,
// whose rows of 7 and 19 entries alternate, uses 99 % of its lanes (68 %
// unsorted): 22.3 us with two lanes per row inside its solve, 17.1 so.  One
// stage per warp; 16 or more warps per SM overlap one another.  x is gathered
// through L1, adjacent rows mostly at adjacent columns.
constexpr int C1_ROWS = 64;

inline size_t c1_smem_bytes(int capb) {
  const size_t b = 64 + (size_t)WTMA_WARPS * (tma_vbytes<double, 1>(capb) + tma_cbytes(capb));
  return b > SUM_SMEM ? b : SUM_SMEM;
}

template <bool DOT>
__global__ void __launch_bounds__(WTMA_WARPS * 32)
    k_csr_f64(const SolveCtl *__restrict__ ctl, int32_t n, const uint32_t *__restrict__ rowptr,
              const uint32_t *__restrict__ colidx, const double *__restrict__ vals,
              const double *__restrict__ x, double *__restrict__ y, double *__restrict__ part,
              int capb, int *err) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ uint32_t keys[WTMA_WARPS][C1_ROWS];
  pdl_wait_and_release();
  if (ctl && ctl->status != ST_RUNNING) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr unsigned FULL = 0xffffffffu;
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm) + warp;
  const size_t vbytes = tma_vbytes<double, 1>(capb);
  unsigned char *base = sm + 64 + (size_t)warp * (vbytes + tma_cbytes(capb));
  double *vb = reinterpret_cast<double *>(base);
  uint32_t *cb = reinterpret_cast<uint32_t *>(base + vbytes), *key = keys[warp];
  if (lane == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
  }
  __syncwarp();
  const int64_t ntiles = ((int64_t)n + C1_ROWS - 1) / C1_ROWS;
  const int64_t nw = (int64_t)gridDim.x * WTMA_WARPS;
  int64_t tile = (int64_t)blockIdx.x * WTMA_WARPS + warp;
  // copies are rounded up to 16 bytes where the matrix goes on behind them
  const size_t vlim = ((size_t)rowptr[n] * 8) & ~size_t(15);
  const size_t clim = ((size_t)rowptr[n] * 4) & ~size_t(15);
  auto up = [](size_t bytes, size_t lim) { return min((bytes + 15) & ~size_t(15), lim); };
  uint32_t c[3], nx[3] = {0, 0, 0};  // row pointers: value i in lane i % 32 of c[i / 32]
  auto fetch = [&](int64_t t) {
    if (t >= ntiles) return;
#pragma unroll
    for (int j = 0; j < 3; ++j)
      nx[j] = rowptr[min((int64_t)n, t * C1_ROWS + min(C1_ROWS, 32 * j + lane))];
  };
  fetch(tile);
  DotAcc<double> acc;
  uint32_t phase = 0;
  for (; tile < ntiles; tile += nw) {
#pragma unroll
    for (int j = 0; j < 3; ++j) c[j] = nx[j];
    const int64_t r0 = tile * C1_ROWS;
    const uint32_t b0 = __shfl_sync(FULL, c[0], 0), b1 = __shfl_sync(FULL, c[2], 0);
    const bool staged = b1 - b0 <= (uint32_t)capb;
    const size_t vs = staged ? ((size_t)b0 * 8) & ~size_t(15) : 0;
    const size_t cs = staged ? ((size_t)b0 * 4) & ~size_t(15) : 0;
    const size_t ve = max(vs, up((size_t)b1 * 8, vlim)), ce = max(cs, up((size_t)b1 * 4, clim));
    __syncwarp();  // the previous tile's buffers are free
    if (staged && lane == 0) {
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(bar, (uint32_t)(ve - vs + (ce - cs)));
      if (ve > vs)
        bulk_g2s(vb, reinterpret_cast<const unsigned char *>(vals) + vs, (uint32_t)(ve - vs), bar);
      if (ce > cs)
        bulk_g2s(cb, reinterpret_cast<const unsigned char *>(colidx) + cs, (uint32_t)(ce - cs), bar);
    }
    fetch(tile + nw);
    // keys: row length (short rows first) | row, rows lane and 32 + lane
    uint32_t ea = __shfl_down_sync(FULL, c[0], 1), eb = __shfl_down_sync(FULL, c[1], 1);
    const uint32_t c1 = __shfl_sync(FULL, c[1], 0);
    if (lane == 31) {
      ea = c1;
      eb = b1;
    }
    uint32_t ka = min(ea - c[0], (1u << 26) - 1) << 6 | lane;
    uint32_t kb = min(eb - c[1], (1u << 26) - 1) << 6 | (32 + lane);
    const uint32_t k0 = __shfl_sync(FULL, ka, 0);
    uint32_t diff = __reduce_or_sync(FULL, (ka ^ k0) | (kb ^ k0)) & ~63u;
    const unsigned below = (1u << lane) - 1u;
    for (; diff; diff &= diff - 1) {
      const uint32_t bit = diff & (0u - diff);
      const unsigned ma = __ballot_sync(FULL, ka & bit), mb = __ballot_sync(FULL, kb & bit);
      const int za = 32 - __popc(ma), z = za + 32 - __popc(mb);
      const int oa = __popc(ma & below), ob = __popc(mb & below);
      key[ka & bit ? z + oa : lane - oa] = ka;
      key[kb & bit ? z + 32 - za + ob : za + lane - ob] = kb;
      __syncwarp();
      ka = key[lane];
      kb = key[32 + lane];
      __syncwarp();
    }
    if (staged) {
      const bool ok = __all_sync(FULL, mbar_wait(bar, phase));
      if (!ok) {
        if (lane == 0) {
          atomicCAS(err, 0, 6 /* DEV_TMA_TIMEOUT */);
          if (!mbar_wait(bar, phase)) atomicExch(err, 8 /* DEV_TMA_UNDRAINED */);
        }
        break;
      }
      phase ^= 1u;
      if ((size_t)b1 * 8 > ve || (size_t)b1 * 4 > ce) {  // the matrix's end: unaligned tails
        if (ve / 8 + lane < b1) vb[(ve - vs) / 8 + lane] = vals[ve / 8 + lane];
        if (ce / 4 + lane < b1) cb[(ce - cs) / 4 + lane] = colidx[ce / 4 + lane];
        __syncwarp();
      }
    }
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      const int i = (int)((pass ? kb : ka) & 63u), j = i + 1;
      const uint32_t s0 = __shfl_sync(FULL, c[0], i & 31), s1 = __shfl_sync(FULL, c[1], i & 31);
      const uint32_t e0 = __shfl_sync(FULL, c[0], j & 31), e1 = __shfl_sync(FULL, c[1], j & 31);
      const uint32_t rb = i < 32 ? s0 : s1, re = j < 32 ? e0 : j < 64 ? e1 : b1;
      if (staged)
        csr_row_f64<DOT>(r0 + i, r0 + i < n, rb, re, vb, cb, vs / 8, cs / 4, x, y, acc);
      else
        csr_row_f64<DOT>(r0 + i, r0 + i < n, rb, re, vals, colidx, 0, 0, x, y, acc);
    }
  }
  if (DOT) {  // CG K1: the last CTA leaves the p.q total in ctl->pq_tot
    const double v = acc.value();
    double t, tot;
    block_sums<1>(&v, &t, sum_buf(sm));
    SolveCtl *s = const_cast<SolveCtl *>(ctl);
    if (finalize_partials<1>(&t, part, &s->tick1, &tot, sum_buf(sm)) && threadIdx.x == 0)
      s->pq_tot = tot;
  }
}

}  // namespace sg

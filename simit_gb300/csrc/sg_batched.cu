// Batched solves of many independent 3x3-blocked systems in one launch.
//
// The systems (e.g. 256 cloth sheets of uneven sizes) are concatenated into
// one block-diagonal matrix: system s owns block rows [sys_ptr[s],
// sys_ptr[s+1]) and its rows reference only its own columns.  A persistent
// kernel runs one whole PCG per CTA: CTAs take systems from a queue ordered
// largest first (longest-processing-time scheduling), and every phase of an
// iteration (SpMV, update, direction) is separated by __syncthreads only —
// systems never share data, so no grid-wide synchronisation exists.  The
// iteration is mixed precision: FP32 matrix and vectors, FP64 dot products,
// 3x3 block-Jacobi preconditioner; convergence (||r|| <= tol ||b||) is
// confirmed on the true residual b - A x accumulated in FP64, and a failed
// confirmation replaces r by it.  Every loop is bounded by maxiters.
//
// Two schedules (the caller's configuration, which the host runtime picks by
// timing them on the batch):
//   - one CTA per system at a time, as above: no grid-wide synchronisation,
//     but a system's iterations run at one SM's bandwidth and a batch whose
//     largest system exceeds its share of the SMs waits for it;
//   - the whole grid on all systems at once (k_batched_grid): every CTA owns
//     an equal run of rows, whichever systems they belong to, and the phases
//     of one iteration of all systems are separated by grid barriers.
//
// The reference solves each mesh with its own Simit program run (one harness
// kernel and a child kernel per loop, src/backend/gpu/gpu_function.cpp:
// 926-951); batching has no counterpart there.
#include <math.h>

#include <vector>

#include "sg_internal.cuh"
#include "sg_solver_kernels.cuh"
#include "sg_spmv_tma.cuh"
#include "sg_tma.cuh"

namespace sg {
namespace {

struct BatchArgs {
  int32_t nsys;
  const int32_t *sys_ptr;   // [nsys+1] block-row ranges
  const int32_t *order;     // [nsys] systems, largest first
  const uint32_t *rowptr, *colidx;
  const float *vals;
  const float *b;           // [n*3]
  float *x;                 // [n*3] in: guess, out: solution
  float *r, *p, *q, *z, *dinv;
  int *queue;               // work counter (zeroed before launch)
  int32_t *iters, *status;  // [nsys]
  double *relres;           // [nsys]
  double tol;
  int maxiters;
};

template <int G>
__device__ __forceinline__ double cta_sum(double v, double *sh) {
  // fixed-order block reduction (blockDim.x <= 1024)
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = (threadIdx.x < (blockDim.x >> 5)) ? sh[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) sh[32] = t;
  }
  __syncthreads();
  return sh[32];
}

// y = A x on rows [r0, r1) (G lanes per row); optional FP64 true residual
// y = b - A x accumulated in FP64 (x FP32) with partial of ||y||^2.
template <int G>
__device__ __forceinline__ double cta_spmv(const BatchArgs &a, int r0, int r1, const float *xv,
                                           float *y, bool residual, double *rr_out) {
  const int gl = threadIdx.x & (G - 1);
  const unsigned mask = group_mask<G>();
  const int groups = blockDim.x / G;
  double acc = 0;
  for (int r = r0 + (int)(threadIdx.x / G); r < r1; r += groups) {
    const uint32_t e = a.rowptr[r + 1];
    if (residual) {  // FP64 accumulation (the true residual)
      double s0 = 0, s1 = 0, s2 = 0;
      for (uint32_t q = a.rowptr[r] + gl; q < e; q += G) {
        const uint32_t c = a.colidx[q];
        const float *v = a.vals + (size_t)q * 9;
        const float x0 = xv[c * 3], x1 = xv[c * 3 + 1], x2 = xv[c * 3 + 2];
        s0 += (double)v[0] * x0 + (double)v[1] * x1 + (double)v[2] * x2;
        s1 += (double)v[3] * x0 + (double)v[4] * x1 + (double)v[5] * x2;
        s2 += (double)v[6] * x0 + (double)v[7] * x1 + (double)v[8] * x2;
      }
      s0 = group_sum<G>(s0, mask);
      s1 = group_sum<G>(s1, mask);
      s2 = group_sum<G>(s2, mask);
      if (gl < 3) {
        const double val = (double)a.b[r * 3 + gl] - (gl == 0 ? s0 : (gl == 1 ? s1 : s2));
        acc += val * val;
        y[r * 3 + gl] = (float)val;
      }
    } else {  // the iteration's SpMV: FP32, as the single-system solver
      float s0 = 0, s1 = 0, s2 = 0;
      for (uint32_t q = a.rowptr[r] + gl; q < e; q += G) {
        const uint32_t c = a.colidx[q];
        const float *v = a.vals + (size_t)q * 9;
        const float x0 = xv[c * 3], x1 = xv[c * 3 + 1], x2 = xv[c * 3 + 2];
        s0 += v[0] * x0 + v[1] * x1 + v[2] * x2;
        s1 += v[3] * x0 + v[4] * x1 + v[5] * x2;
        s2 += v[6] * x0 + v[7] * x1 + v[8] * x2;
      }
      s0 = group_sum<G>(s0, mask);
      s1 = group_sum<G>(s1, mask);
      s2 = group_sum<G>(s2, mask);
      if (gl < 3) y[r * 3 + gl] = gl == 0 ? s0 : (gl == 1 ? s1 : s2);
    }
  }
  if (rr_out) *rr_out = acc;
  return acc;
}

// Inverse of vertex v's diagonal block (its diagonal's where it is singular).
__device__ __forceinline__ void batch_diag_inv(const BatchArgs &a, int v) {
  uint32_t lo = a.rowptr[v], hi = a.rowptr[v + 1];
  const uint32_t end = hi;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a.colidx[mid] < (uint32_t)v) lo = mid + 1; else hi = mid;
  }
  float *D = a.dinv + (size_t)v * 9;
  if (lo >= end || a.colidx[lo] != (uint32_t)v) {
    for (int k = 0; k < 9; ++k) D[k] = 0.f;
    return;
  }
  const float *m = a.vals + (size_t)lo * 9;
  const double c00 = (double)m[4] * m[8] - (double)m[5] * m[7];
  const double c01 = (double)m[5] * m[6] - (double)m[3] * m[8];
  const double c02 = (double)m[3] * m[7] - (double)m[4] * m[6];
  const double det = m[0] * c00 + m[1] * c01 + m[2] * c02;
  if (!(fabs(det) > 0.0)) {
    for (int k = 0; k < 9; ++k) D[k] = 0.f;
    for (int k = 0; k < 3; ++k) D[k * 4] = m[k * 4] != 0.f ? 1.f / m[k * 4] : 0.f;
    return;
  }
  const double id = 1.0 / det;
  D[0] = (float)(c00 * id);
  D[1] = (float)(((double)m[2] * m[7] - (double)m[1] * m[8]) * id);
  D[2] = (float)(((double)m[1] * m[5] - (double)m[2] * m[4]) * id);
  D[3] = (float)(c01 * id);
  D[4] = (float)(((double)m[0] * m[8] - (double)m[2] * m[6]) * id);
  D[5] = (float)(((double)m[2] * m[3] - (double)m[0] * m[5]) * id);
  D[6] = (float)(c02 * id);
  D[7] = (float)(((double)m[1] * m[6] - (double)m[0] * m[7]) * id);
  D[8] = (float)(((double)m[0] * m[4] - (double)m[1] * m[3]) * id);
}

template <int G>
__global__ void k_batched_pcg(BatchArgs a) {
  __shared__ double sh[34];
  __shared__ int sys_sh;
  for (;;) {
    if (threadIdx.x == 0) {
      const int k = atomicAdd(a.queue, 1);
      sys_sh = k < a.nsys ? a.order[k] : -1;
    }
    __syncthreads();
    const int s = sys_sh;
    __syncthreads();
    if (s < 0) break;
    const int r0 = a.sys_ptr[s], r1 = a.sys_ptr[s + 1];
    const int i0 = r0 * 3, i1 = r1 * 3;
    // block-Jacobi inverse of the diagonal blocks
    for (int v = r0 + threadIdx.x; v < r1; v += blockDim.x) batch_diag_inv(a, v);
    // b'b
    double bb = 0;
    for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) bb += (double)a.b[i] * a.b[i];
    bb = cta_sum<G>(bb, sh);
    const double tol2 = a.tol * a.tol * bb;
    // r = b - A x (FP64 accumulation)
    double rr = 0;
    cta_spmv<G>(a, r0, r1, a.x, a.r, true, &rr);
    rr = cta_sum<G>(rr, sh);
    int it = 0, st = 0;
    double rz = 0;
    auto precondition = [&]() {
      DotAcc<float> t;
      for (int v = r0 + threadIdx.x; v < r1; v += blockDim.x) {
        const float *D = a.dinv + (size_t)v * 9;
        const float q0 = a.r[v * 3], q1 = a.r[v * 3 + 1], q2 = a.r[v * 3 + 2];
        for (int k = 0; k < 3; ++k) {
          const float zk = D[k * 3] * q0 + D[k * 3 + 1] * q1 + D[k * 3 + 2] * q2;
          a.z[v * 3 + k] = zk;
          t.add(a.r[v * 3 + k], zk);
        }
      }
      return cta_sum<G>(t.value(), sh);
    };
    if (!(rr > tol2)) {
      st = SG_STATUS_CONVERGED;
    } else {
      rz = precondition();
      for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) a.p[i] = a.z[i];
      __syncthreads();
    }
    while (!st) {
      if (it >= a.maxiters) {
        st = SG_STATUS_MAXITER;
        break;
      }
      // q = A p, p.q
      cta_spmv<G>(a, r0, r1, a.p, a.q, false, nullptr);
      __syncthreads();
      DotAcc<float> pqa;
      for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) pqa.add(a.p[i], a.q[i]);
      const double pq = cta_sum<G>(pqa.value(), sh);
      if (!(pq > 0.0) || !isfinite(pq)) {
        st = isfinite(pq) ? SG_STATUS_BREAKDOWN : SG_STATUS_NAN;
        break;
      }
      const float al = (float)(rz / pq);
      DotAcc<float> rra;
      for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
        a.x[i] += al * a.p[i];
        const float ri = a.r[i] - al * a.q[i];
        a.r[i] = ri;
        rra.add(ri, ri);
      }
      const double rrl = cta_sum<G>(rra.value(), sh);
      ++it;
      double rznew = precondition();
      if (rrl <= tol2) {
        // confirm on the true residual; replace r by it when it fails
        double rt = 0;
        __syncthreads();
        cta_spmv<G>(a, r0, r1, a.x, a.r, true, &rt);
        rt = cta_sum<G>(rt, sh);
        rr = rt;
        if (rt <= tol2) {
          st = SG_STATUS_CONVERGED;
          break;
        }
        rznew = precondition();
      }
      if (!isfinite(rznew)) {
        st = SG_STATUS_NAN;
        break;
      }
      const float be = (float)(rznew / rz);
      rz = rznew;
      for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) a.p[i] = a.z[i] + be * a.p[i];
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      a.iters[s] = it;
      a.status[s] = st;
      a.relres[s] = bb > 0 ? sqrt(rr / bb) : 0.0;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// The whole grid on all systems
// ---------------------------------------------------------------------------
// The rows of every system are cut into chunks of GB_C; CTA b of NB owns the
// chunks [T b / NB, T (b+1) / NB), so a CTA meets a few systems (segments)
// and a system a few CTAs.  An iteration of all systems is three phases with
// a grid barrier after each: q = A p and p.q; r, z and r.r, r.z; x, p.  A
// segment's dot products go to part[k][b + s] (b + s grows by at least one
// from segment to segment, and a system's segments are consecutive); after
// the barrier every CTA that holds rows of a system sums them in the same
// order and takes the same decision.  k: a DotSlot; no slot is read and written
// between two barriers, or a CTA that is ahead would overwrite what one behind
// has still to read (b.b shared the slot of r.r, which the first pass writes
// right after b.b's sum).  A system whose iterated residual passes
// spends the first phase of the next GB_K passes on its true residual, a part
// in each (CONFIRM): FP64 work that only its own CTAs share would otherwise
// make one pass four times as long for every system.
//
// The arithmetic of a row, a vertex and a decision is k_batched_pcg's; the
// dot products differ by the order of their FP64 sums.
//
// Bound by memory: an iteration streams the matrix (40 bytes a block) and 40
// floats a vertex of vectors and inverse blocks.  What keeps it near that:
//   - a warp's tiles (GB_R rows of every chunk) arrive by bulk copies into
//     two stages, and the row pointers of the tile after next are loaded
//     before the current one is computed, so that no tile waits for a chain
//     of loads (5,600 cycles a tile when it did, 1.9 times the time);
//   - p is kept as four floats a vertex, one load a gather instead of three;
//   - the polls of the grid barrier are relaxed loads: an acquire each would
//     empty the SM's L1 under the CTA that still works.
// 96 sheets of 32..256 vertices a side (2.2 million vertices, 130 iterations):
// 49 ms, 255 with one CTA a system; a pass is 0.36 ms, 0.28 of it the product
// at 3.6 TB/s.  2 sheets of 16..48: 2.3 ms, 7.1.  300 sheets of 8..24: 4.9 ms,
// where one CTA a system takes 4.0 (19 us a pass is barriers and latency).
constexpr int GB_T = 256, GB_W = GB_T / 32;
constexpr int GB_C = 64;            // rows per chunk
constexpr int GB_R = GB_C / GB_W;   // rows per warp tile
constexpr int GB_ST = 2;            // bulk-copy stages of a warp
constexpr int GB_SEG = 16;          // segments kept in shared memory
constexpr int GB_K = 4;             // passes a confirmation is spread over
constexpr int GB_MAXSMEM = 220 * 1024;
enum GridState : int { GS_RUN = 0, GS_CONFIRM = 1, GS_DONE = 2 };
// partial sums: b.b (first pass), p.q or the true residual's r.r, r.r, r.z
enum DotSlot : int { DS_BB = 0, DS_PQ = 1, DS_RR = 2, DS_RZ = 3, DS_N = 4 };

struct GridArgs {
  BatchArgs b;
  int64_t nnzb;
  float4 *p;                 // [n] directions
  const int32_t *chunk_ptr;  // [nsys+1] chunks before each system
  double *part;              // [DS_N][nb + nsys]
  unsigned int *bar;         // barrier arrivals (zeroed before launch)
  int *ndone;                // systems finished (zeroed before launch)
  int *err;
  struct Seg *segs;          // [nb + nsys] segments of CTAs that meet more than GB_SEG
  double *wps;               // [nb + nsys][DS_N][GB_W]
  int capb;                  // blocks per warp stage; -1: every tile is read from global memory
};

struct Seg {
  double rz, tol2, bb, rr;
  float al, be;
  int ra, rb;  // rows of the segment
  int st, it, sys, lead, end;
  int sl;  // the confirmation's part of this pass (GB_K: all of it)
};

// chunk_ptr of the systems (one CTA; systems without rows finish here).
__global__ void __launch_bounds__(1024) k_grid_plan(BatchArgs a, int32_t *chunk_ptr, int *ndone) {
  __shared__ int sh[33];
  int base = 0;
  if (threadIdx.x == 0) chunk_ptr[0] = 0;
  for (int s0 = 0; s0 < a.nsys; s0 += 1024) {
    const int s = s0 + (int)threadIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int v = 0;
    if (s < a.nsys) {
      const int rows = a.sys_ptr[s + 1] - a.sys_ptr[s];
      v = (rows + GB_C - 1) / GB_C;
      if (rows <= 0) {
        a.iters[s] = 0;
        a.status[s] = SG_STATUS_CONVERGED;
        a.relres[s] = 0.0;
        atomicAdd(ndone, 1);
        v = 0;
      }
    }
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += t;
    }
    if (lane == 31) sh[w] = v;
    __syncthreads();
    if (w == 0) {
      int t = sh[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += u;
      }
      sh[lane] = t;
    }
    __syncthreads();
    if (s < a.nsys) chunk_ptr[s + 1] = base + v + (w ? sh[w - 1] : 0);
    base += sh[31];
    __syncthreads();
  }
}

// Row r (blocks q0 .. e) of q = A p from its staged (or global) values and
// columns; the lane split and order of cta_spmv.  p was written by other CTAs
// of this launch, so it is read with ordinary loads.
template <int G>
__device__ __forceinline__ void grid_row(int r, uint32_t q0, uint32_t e, int gl, unsigned mask,
                                         const float *vb, const uint32_t *cb, size_t voff,
                                         size_t coff, const float4 *x, float *y,
                                         DotAcc<float> &acc) {
  constexpr int U = (16 + G - 1) / G;  // gathers in flight a lane
  float4 xg[U];
  float a0 = 0.f, a1 = 0.f, a2 = 0.f;
  q0 += gl;
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const uint32_t q = q0 + k * G;
    if (q < e) xg[k] = x[cb[q - coff]];
  }
  auto block = [&](uint32_t q, const float4 &t) {
    const float *v = vb + ((size_t)q * 9 - voff);
    a0 += v[0] * t.x + v[1] * t.y + v[2] * t.z;
    a1 += v[3] * t.x + v[4] * t.y + v[5] * t.z;
    a2 += v[6] * t.x + v[7] * t.y + v[8] * t.z;
  };
#pragma unroll
  for (int k = 0; k < U; ++k)
    if (q0 + k * G < e) block(q0 + k * G, xg[k]);
  for (uint32_t q = q0 + U * G; q < e; q += G) block(q, x[cb[q - coff]]);
  a0 = group_sum<G>(a0, mask);
  a1 = group_sum<G>(a1, mask);
  a2 = group_sum<G>(a2, mask);
  if (gl < 3) {
    const float yv = gl == 0 ? a0 : (gl == 1 ? a1 : a2);
    y[(size_t)r * 3 + gl] = yv;
    acc.add(reinterpret_cast<const float *>(x + r)[gl], yv);
  }
}

template <int G>
__device__ __noinline__ DotAcc<float> grid_row_global(int r, uint32_t q0, uint32_t e, int gl,
                                                      unsigned mask, const float *vals,
                                                      const uint32_t *cols, const float4 *x,
                                                      float *y, DotAcc<float> acc) {
  grid_row<G>(r, q0, e, gl, mask, vals, cols, 0, 0, x, y, acc);
  return acc;
}

// Row r of r = b - A x with FP64 accumulation; the lane's part of ||r||^2.
// The entries are widened by integer operations: a conversion costs the FP64
// pipe as much as a multiply-add.  (Not inlined: it runs twice a solve, and
// its registers would spill the iteration's.)
template <int G>
__device__ __noinline__ double grid_residual_row(int r, uint32_t q0, uint32_t e, int gl,
                                                    unsigned mask, const float *vb,
                                                    const uint32_t *cb, size_t voff, size_t coff,
                                                    const float *x, const float *b, float *y) {
  double s0 = 0, s1 = 0, s2 = 0;
#pragma unroll 2
  for (uint32_t q = q0 + gl; q < e; q += G) {
    const float *v = vb + ((size_t)q * 9 - voff), *xc = x + (size_t)cb[q - coff] * 3;
    const double x0 = widen_f32(xc[0]), x1 = widen_f32(xc[1]), x2 = widen_f32(xc[2]);
    s0 = fma(widen_f32(v[2]), x2, fma(widen_f32(v[1]), x1, fma(widen_f32(v[0]), x0, s0)));
    s1 = fma(widen_f32(v[5]), x2, fma(widen_f32(v[4]), x1, fma(widen_f32(v[3]), x0, s1)));
    s2 = fma(widen_f32(v[8]), x2, fma(widen_f32(v[7]), x1, fma(widen_f32(v[6]), x0, s2)));
  }
  s0 = group_sum<G>(s0, mask);
  s1 = group_sum<G>(s1, mask);
  s2 = group_sum<G>(s2, mask);
  if (gl >= 3) return 0.0;
  const double val = (double)b[r * 3 + gl] - (gl == 0 ? s0 : (gl == 1 ? s1 : s2));
  y[r * 3 + gl] = (float)val;
  return val * val;
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

template <int G>
__global__ void __launch_bounds__(GB_T, 2) k_batched_grid(GridArgs g) {
  extern __shared__ __align__(16) unsigned char gsm[];
  __shared__ int ok_sh, stop_sh, ns_sh, lo_sh;
  const BatchArgs &a = g.b;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = gridDim.x, b = blockIdx.x;
  const int cap = max(g.capb, 0);
  const size_t vbytes = tma_vbytes<float>(cap), stage = vbytes + tma_cbytes(cap);
  Seg *seg = reinterpret_cast<Seg *>(gsm);
  double *wp = reinterpret_cast<double *>(seg + GB_SEG);  // [segment][DS_N][GB_W]
  unsigned char *raw = reinterpret_cast<unsigned char *>(wp + GB_SEG * DS_N * GB_W);
  uint64_t *bar = reinterpret_cast<uint64_t *>(raw) + warp * GB_ST;
  unsigned char *base = raw + GB_W * GB_ST * 8 + (size_t)warp * GB_ST * stage;
  if (lane == 0) {
    for (int k = 0; k < GB_ST; ++k) mbar_init(&bar[k], 1);
    mbar_fence_init();
  }
  // the CTA's chunks and segments
  const int64_t T = g.chunk_ptr[a.nsys];
  const int c0 = (int)(T * b / nb), c1 = (int)(T * (b + 1) / nb);
  if (warp == 0) {
    // pass 0 counts the segments, pass 1 writes them: to shared memory, or
    // to the CTA's part of the global list (from b + its first system on)
    int ns_ = 0, lo = 0;
    if (c0 < c1) {
      int hi = a.nsys - 1;  // the last system that starts at or before chunk c0
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (g.chunk_ptr[mid] <= c0) lo = mid; else hi = mid - 1;
      }
      for (int pass = 0; pass < 2; ++pass) {
        if (pass && ns_ > GB_SEG) {
          seg = g.segs + b + lo;
          wp = g.wps + ((size_t)b + lo) * DS_N * GB_W;
        }
        ns_ = 0;
        for (int s0 = lo; s0 < a.nsys && g.chunk_ptr[s0] < c1; s0 += 32) {
          const int s = s0 + lane;
          int k0 = c1, k1 = c1;
          if (s < a.nsys) {
            k0 = g.chunk_ptr[s];
            k1 = g.chunk_ptr[s + 1];
          }
          const bool mine = k0 < k1 && k0 < c1 && k1 > c0;  // (no system without rows)
          const unsigned m = __ballot_sync(0xffffffffu, mine);
          if (pass && mine) {
            const int r0 = a.sys_ptr[s], r1 = a.sys_ptr[s + 1];
            Seg q = {};
            q.sys = s;
            q.ra = r0 + (max(k0, c0) - k0) * GB_C;
            q.rb = k1 <= c1 ? r1 : r0 + (c1 - k0) * GB_C;
            q.lead = k0 >= c0;
            q.st = GS_CONFIRM;  // the first pass computes r = b - A x
            q.sl = GB_K;
            seg[ns_ + __popc(m & ((1u << lane) - 1u))] = q;
          }
          ns_ += __popc(m);
        }
      }
    }
    if (lane == 0) {
      ns_sh = ns_;
      lo_sh = lo;
    }
  }
  __syncthreads();
  const int ns = ns_sh;
  if (ns > GB_SEG) {
    seg = g.segs + b + lo_sh;
    wp = g.wps + ((size_t)b + lo_sh) * DS_N * GB_W;
  }
  const int64_t np = (int64_t)nb + a.nsys;
  unsigned int arrived = 0;
  // a segment's partial sums kb .. ke-1, from the warps' in wp
  auto publish = [&](int kb, int ke) {
    __syncthreads();
    for (int t = tid; t < ns * (ke - kb); t += GB_T) {
      const int j = t / (ke - kb), k = kb + t % (ke - kb);
      if (seg[j].st == GS_DONE) continue;
      double v = 0;
      for (int w = 0; w < GB_W; ++w) v += wp[(j * DS_N + k) * GB_W + w];
      g.part[k * np + b + seg[j].sys] = v;
    }
  };
  auto sync_grid = [&]() {
    arrived += nb;
    return grid_barrier(g.bar, arrived, g.err, &ok_sh);
  };
  // sum of partial k over the system's segments (all CTAs in the same order)
  auto total = [&](int s, int k) {
    const int64_t k0 = g.chunk_ptr[s], k1 = (int64_t)g.chunk_ptr[s + 1] - 1;
    const int b0 = (int)(((k0 + 1) * nb - 1) / T), b1 = (int)(((k1 + 1) * nb - 1) / T);
    double v = 0;
    for (int i = b0 + lane; i <= b1; i += 32)
      if ((int)(T * i / nb) < (int)(T * (i + 1) / nb)) v += __ldcg(g.part + k * np + i + s);
    return __shfl_sync(0xffffffffu, warp_sum(v), 0);
  };
  auto finish = [&](Seg &q, int status) {  // one thread per segment
    q.st = GS_DONE;
    if (q.lead) {
      a.iters[q.sys] = q.it;
      a.status[q.sys] = status;
      a.relres[q.sys] = q.bb > 0 ? sqrt(q.rr / q.bb) : 0.0;
      __threadfence();
      atomicAdd(g.ndone, 1);
    }
  };
  // z = M r of one vertex, its r.z
  auto precondition = [&](int v, const float *D, const float *rv, DotAcc<float> &t) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float zk = D[k * 3] * rv[0] + D[k * 3 + 1] * rv[1] + D[k * 3 + 2] * rv[2];
      a.z[v * 3 + k] = zk;
      t.add(rv[k], zk);
    }
  };
  // set-up: inverse diagonal, b'b
  for (int j = 0; j < ns; ++j) {
    const Seg q = seg[j];
    for (int v = q.ra + tid; v < q.rb; v += GB_T) batch_diag_inv(a, v);
    double bb = 0;
    for (int i = q.ra * 3 + tid; i < q.rb * 3; i += GB_T) bb += (double)a.b[i] * a.b[i];
    bb = warp_sum(bb);
    if (lane == 0) wp[(j * DS_N + DS_BB) * GB_W + warp] = bb;
  }

  const int gl = lane & (G - 1);
  const unsigned mask = group_mask<G>();
  const size_t vend = ((size_t)g.nnzb * 36) & ~size_t(15), cend = ((size_t)g.nnzb * 4) & ~size_t(15);
  uint32_t nth = 0;  // tiles this warp has consumed (stage and parity)
  // (a system takes an iteration and a confirmation each, at most)
  for (int64_t pass = 0; pass <= (1 + GB_K) * ((int64_t)a.maxiters + 2); ++pass) {
    __syncthreads();
    if (tid == 0) stop_sh = *(volatile int *)g.ndone >= a.nsys;
    __syncthreads();
    if (stop_sh) break;
    // phase 1: q = A p of the running systems, the true residual of the
    // others
    {
      struct Walk {
        int j, row;
        uint32_t rp;  // lane l: row pointer of row + l (the segment's end at most)
      };
      // the tile after w; j == ns at the end
      auto next = [&](const Walk &w) {
        Walk t = {w.j, w.row + GB_C, 0u};
        if (t.j >= 0 && seg[t.j].st == GS_CONFIRM && seg[t.j].sl < GB_K)
          t.row += (GB_K - 1) * GB_C;  // one chunk in GB_K
        while (t.j < ns && (t.j < 0 || t.row >= seg[t.j].rb || seg[t.j].st == GS_DONE)) {
          if (++t.j == ns) break;
          t.row = seg[t.j].ra + warp * GB_R;
          if (seg[t.j].st == GS_CONFIRM && seg[t.j].sl < GB_K) t.row += seg[t.j].sl * GB_C;
        }
        if (t.j < ns) t.rp = a.rowptr[min(t.row + min(lane, GB_R), seg[t.j].rb)];
        return t;
      };
      // a tile's copies end at the next 16-byte boundary; only at the
      // matrix's end a tail of less than 16 bytes is left for the lanes
      auto issue = [&](const Walk &w, int st) {
        const uint32_t b0 = __shfl_sync(0xffffffffu, w.rp, 0);
        const uint32_t b1 = __shfl_sync(0xffffffffu, w.rp, GB_R);
        if (lane) return;
        const size_t vs = ((size_t)b0 * 36) & ~size_t(15), cs = ((size_t)b0 * 4) & ~size_t(15);
        const size_t ve = min(((size_t)b1 * 36 + 15) & ~size_t(15), vend);
        const size_t ce = min(((size_t)b1 * 4 + 15) & ~size_t(15), cend);
        unsigned char *vb = base + (size_t)st * stage;
        fence_proxy_async_smem();
        if ((int)(b1 - b0) > g.capb) {  // larger than the stage: read from global
          mbar_arrive_expect_tx(&bar[st], 0);
          return;
        }
        const uint32_t vn = ve > vs ? (uint32_t)(ve - vs) : 0u, cn = ce > cs ? (uint32_t)(ce - cs) : 0u;
        mbar_arrive_expect_tx(&bar[st], vn + cn);
        if (vn) bulk_g2s(vb, reinterpret_cast<const unsigned char *>(a.vals) + vs, vn, &bar[st]);
        if (cn)
          bulk_g2s(vb + vbytes, reinterpret_cast<const unsigned char *>(a.colidx) + cs, cn,
                   &bar[st]);
      };
      Walk cur = next(Walk{-1, 0, 0u}), ahead = cur;
      if (cur.j < ns) {
        issue(cur, nth & 1);
        ahead = next(cur);
      }
      DotAcc<float> acc;
      double racc = 0;
      bool ok = true;
      while (cur.j < ns) {
        const int st = nth & 1;
        const bool more = ahead.j < ns;
        Walk far = ahead;
        if (more) {
          issue(ahead, st ^ 1);
          far = next(ahead);
        }
        ok = __all_sync(0xffffffffu, mbar_wait(&bar[st], (nth >> 1) & 1));
        if (!ok) {
          if (lane == 0) {
            atomicCAS(g.err, 0, DEV_TMA_TIMEOUT);
            // the copies in flight land before the CTA leaves
            bool drained = mbar_wait(&bar[st], (nth >> 1) & 1);
            if (more) drained = mbar_wait(&bar[st ^ 1], ((nth + 1) >> 1) & 1) && drained;
            if (!drained) atomicExch(g.err, DEV_TMA_UNDRAINED);
          }
          break;
        }
        ++nth;
        const uint32_t b0 = __shfl_sync(0xffffffffu, cur.rp, 0);
        const uint32_t b1 = __shfl_sync(0xffffffffu, cur.rp, GB_R);
        const bool staged = (int)(b1 - b0) <= g.capb;
        const size_t vs = staged ? ((size_t)b0 * 36) & ~size_t(15) : 0;
        const size_t cs = staged ? ((size_t)b0 * 4) & ~size_t(15) : 0;
        float *vb = reinterpret_cast<float *>(base + (size_t)st * stage);
        uint32_t *cb = reinterpret_cast<uint32_t *>(base + (size_t)st * stage + vbytes);
        if (staged && ((size_t)b1 * 36 > vend || (size_t)b1 * 4 > cend)) {
          const size_t v0 = max(vend, vs) / 4, c0_ = max(cend, cs) / 4;
          if (v0 + lane < (size_t)b1 * 9) vb[v0 + lane - vs / 4] = a.vals[v0 + lane];
          if (c0_ + lane < (size_t)b1) cb[c0_ + lane - cs / 4] = a.colidx[c0_ + lane];
        }
        __syncwarp();
        const bool run = seg[cur.j].st == GS_RUN;
        const int rb = seg[cur.j].rb;
#pragma unroll
        for (int pp = 0; pp < GB_R * G / 32; ++pp) {
          const int rl = pp * (32 / G) + lane / G, r = cur.row + rl;
          const uint32_t q0 = __shfl_sync(0xffffffffu, cur.rp, rl);
          const uint32_t e = __shfl_sync(0xffffffffu, cur.rp, rl + 1);
          if (r < rb) {
            if (run) {
              if (staged)
                grid_row<G>(r, q0, e, gl, mask, vb, cb, vs / 4, cs / 4, g.p, a.q, acc);
              else
                acc = grid_row_global<G>(r, q0, e, gl, mask, a.vals, a.colidx, g.p, a.q, acc);
            } else {
              racc += grid_residual_row<G>(r, q0, e, gl, mask, staged ? vb : a.vals,
                                           staged ? cb : a.colidx, vs / 4, cs / 4, a.x, a.b, a.r);
            }
          }
        }
        __syncwarp();
        const int j = cur.j;
        if (!more || ahead.j != j) {  // the segment's last tile of this warp
          const double t = warp_sum(run ? acc.value() : racc);
          if (lane == 0) wp[(j * DS_N + DS_PQ) * GB_W + warp] = t;
          acc = DotAcc<float>();
          racc = 0;
        }
        if (!more) break;
        cur = ahead;
        ahead = far;
      }
      if (__syncthreads_or(!ok)) return;
      // a warp without a tile in a segment has not set its sum
      for (int j = 0; j < ns; ++j) {
        const int skip = seg[j].st == GS_CONFIRM && seg[j].sl < GB_K ? seg[j].sl : 0;
        if (lane == 0 && seg[j].ra + skip * GB_C + warp * GB_R >= seg[j].rb)
          wp[(j * DS_N + DS_PQ) * GB_W + warp] = 0.0;
      }
    }
    publish(pass == 0 ? DS_BB : DS_PQ, DS_PQ + 1);
    if (!sync_grid()) return;
    // phase 2: alpha; r and z of the running systems, z of the others that
    // have not converged
    for (int j = warp; j < ns; j += GB_W) {
      if (seg[j].st == GS_DONE) continue;
      const double t = total(seg[j].sys, DS_PQ);
      const double bb = pass == 0 ? total(seg[j].sys, DS_BB) : 0.0;
      if (lane == 0) {
        Seg &q = seg[j];
        if (pass == 0) {
          q.bb = bb;
          q.tol2 = a.tol * a.tol * bb;
        }
        q.al = 0.f;
        if (q.st == GS_RUN) {
          if (!(t > 0.0) || !isfinite(t))
            finish(q, isfinite(t) ? SG_STATUS_BREAKDOWN : SG_STATUS_NAN);
          else
            q.al = (float)(q.rz / t);
        } else {
          q.rr = q.sl == 0 || q.sl == GB_K ? t : q.rr + t;
          q.sl = q.sl < GB_K ? q.sl + 1 : GB_K;
          if (q.sl == GB_K) {  // the whole residual
            if (pass == 0 ? !(q.rr > q.tol2) : q.rr <= q.tol2) finish(q, SG_STATUS_CONVERGED);
            else if (pass == 0 && a.maxiters <= 0) finish(q, SG_STATUS_MAXITER);
          }
        }
      }
    }
    __syncthreads();
    for (int j = 0; j < ns; ++j) {
      const Seg q = seg[j];
      if (q.st == GS_DONE || (q.st == GS_CONFIRM && q.sl < GB_K)) continue;
      DotAcc<float> rra, t;
      // two vertices a thread at a time, their loads before the first store
      for (int v0 = q.ra + tid; v0 < q.rb; v0 += 2 * GB_T) {
        float rv[2][3], qv[2][3], D[2][9];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int v = v0 + u * GB_T;
          if (v < q.rb) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              rv[u][k] = a.r[v * 3 + k];
              qv[u][k] = a.q[v * 3 + k];
            }
#pragma unroll
            for (int k = 0; k < 9; ++k) D[u][k] = a.dinv[(size_t)v * 9 + k];
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int v = v0 + u * GB_T;
          if (v < q.rb) {
            if (q.st == GS_RUN) {
#pragma unroll
              for (int k = 0; k < 3; ++k) {
                rv[u][k] = rv[u][k] - q.al * qv[u][k];
                a.r[v * 3 + k] = rv[u][k];
                rra.add(rv[u][k], rv[u][k]);
              }
            }
            precondition(v, D[u], rv[u], t);
          }
        }
      }
      const double s_rr = warp_sum(rra.value()), s_rz = warp_sum(t.value());
      if (lane == 0) {
        wp[(j * DS_N + DS_RR) * GB_W + warp] = s_rr;
        wp[(j * DS_N + DS_RZ) * GB_W + warp] = s_rz;
      }
    }
    publish(DS_RR, DS_RZ + 1);
    if (!sync_grid()) return;
    // phase 3: the decision; x and p
    for (int j = warp; j < ns; j += GB_W) {
      if (seg[j].st == GS_DONE || (seg[j].st == GS_CONFIRM && seg[j].sl < GB_K)) continue;
      const double rr = total(seg[j].sys, DS_RR), rz = total(seg[j].sys, DS_RZ);
      if (lane == 0) {
        Seg &q = seg[j];
        bool turn = true;  // a new direction
        if (q.st == GS_RUN) {
          ++q.it;
          turn = !(rr <= q.tol2);
        } else {
          q.al = 0.f;
        }
        q.be = 0.f;
        if (turn) {
          if (pass > 0) q.be = (float)(rz / q.rz);
          q.rz = rz;
          q.st = GS_RUN;
        } else {
          q.st = GS_CONFIRM;
          q.sl = 0;
        }
        q.end = turn && !isfinite(rz);  // after this x
      }
    }
    __syncthreads();
    for (int j = 0; j < ns; ++j) {
      const Seg q = seg[j];
      if (q.st == GS_DONE || (q.st == GS_CONFIRM && q.al == 0.f)) continue;
      const bool newp = q.st == GS_RUN;
      // two vertices a thread at a time, their loads before the first store
      for (int v0 = q.ra + tid; v0 < q.rb; v0 += 2 * GB_T) {
        float4 pv[2];
        float xv[2][3], zv[2][3];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int v = v0 + u * GB_T;
          if (v < q.rb) {
            if (pass > 0) pv[u] = g.p[v];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              xv[u][k] = a.x[v * 3 + k];
              zv[u][k] = a.z[v * 3 + k];
            }
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int v = v0 + u * GB_T;
          if (v < q.rb) {
            if (pass == 0) {
              g.p[v] = make_float4(zv[u][0], zv[u][1], zv[u][2], 0.f);
              continue;
            }
            if (q.al != 0.f) {
              a.x[v * 3] = xv[u][0] + q.al * pv[u].x;
              a.x[v * 3 + 1] = xv[u][1] + q.al * pv[u].y;
              a.x[v * 3 + 2] = xv[u][2] + q.al * pv[u].z;
            }
            if (newp)
              g.p[v] = make_float4(zv[u][0] + q.be * pv[u].x, zv[u][1] + q.be * pv[u].y,
                                   zv[u][2] + q.be * pv[u].z, 0.f);
          }
        }
      }
    }
    __syncthreads();
    for (int j = tid; j < ns; j += GB_T) {
      Seg &q = seg[j];
      if (q.st == GS_DONE) continue;
      if (q.end) finish(q, SG_STATUS_NAN);
      else if (q.st == GS_RUN && q.it >= a.maxiters) finish(q, SG_STATUS_MAXITER);
    }
    if (!sync_grid()) return;
  }
}

// Lanes per row, threads per CTA; threads 0: the whole grid on all systems.
struct BatchCfg {
  int G, threads;
};
const BatchCfg kCfgs[] = {{4, 512}, {8, 512}, {4, 1024}, {8, 1024}, {4, 256}, {8, 256},
                          {4, 0},   {8, 0}};
constexpr int kNumCfgs = sizeof(kCfgs) / sizeof(kCfgs[0]);

// Grid and shared memory of the grid-wide kernel for n rows of nnzb blocks
// in nsys systems.
constexpr int GB_MAXCTAS = 2;  // CTAs an SM (the kernel's launch bounds)
template <int G>
int grid_config(Ctx *c, int32_t n, int64_t nnzb, int nsys, bool aligned, int *grid, int *capb,
                size_t *smem) {
  // room for a tile 15 % above the average (every byte of the stages comes off
  // the L1 that the gathers live in: stages of a third above cost 10 %);
  // larger ones are read from global memory.  Bulk copies start on 16-byte
  // boundaries, so a matrix that does not is read from global memory throughout
  int cap = (int)((double)nnzb / n * GB_R * 1.15) + 6;
  if (cap > 256) cap = 256;
  if (!aligned) cap = 0;
  *capb = aligned ? cap : -1;
  auto kern = k_batched_grid<G>;
  static PerDeviceOnce attr;
  SG_TRY(once_per_device(attr, c->device, [&]() -> int {
    SG_CHECK_CUDA(
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GB_MAXSMEM));
    return SG_OK;
  }));
  *smem = GB_SEG * (sizeof(Seg) + DS_N * GB_W * 8) + GB_W * GB_ST * 8 +
          (size_t)GB_W * GB_ST * (tma_vbytes<float>(cap) + tma_cbytes(cap));
  int per_sm = 0;
  SG_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, GB_T, *smem));
  if (per_sm > GB_MAXCTAS) per_sm = GB_MAXCTAS;
  int64_t gsz = (int64_t)per_sm * c->num_sms;
  const int64_t chunks = (int64_t)n / GB_C + nsys;       // at most
  if (gsz > (chunks + 1) / 2) gsz = (chunks + 1) / 2;  // two chunks a CTA at least
  *grid = (int)gsz;
  return SG_OK;
}

// Scratch of the grid-wide kernel.
struct GridScratch {
  float4 *p;
  double *part, *wps;
  Seg *segs;
  int32_t *chunk_ptr;
  unsigned int *bar;
};

int launch(Ctx *c, cudaStream_t st, const BatchArgs &a, int cfg, int32_t n, int64_t nnzb,
           const GridScratch &w) {
  const BatchCfg &k = kCfgs[cfg];
  if (k.threads == 0) {
    GridArgs g;
    int grid = 0;
    size_t smem = 0;
    const bool al = (uintptr_t)a.vals % 16 == 0 && (uintptr_t)a.colidx % 16 == 0;
    SG_TRY(k.G == 4 ? grid_config<4>(c, n, nnzb, a.nsys, al, &grid, &g.capb, &smem)
                    : grid_config<8>(c, n, nnzb, a.nsys, al, &grid, &g.capb, &smem));
    SG_REQUIRE(grid >= 1, "sg_batched_pcg: the grid-wide kernel does not fit an SM");
    g.b = a;
    g.nnzb = nnzb;
    g.p = w.p;
    g.chunk_ptr = w.chunk_ptr;
    g.part = w.part;
    g.segs = w.segs;
    g.wps = w.wps;
    g.bar = w.bar;
    g.ndone = (int *)w.bar + 1;
    g.err = c->d_err;
    SG_CHECK_CUDA(cudaMemsetAsync(w.bar, 0, 2 * sizeof(int), st));
    k_grid_plan<<<1, 1024, 0, st>>>(a, w.chunk_ptr, g.ndone);
    SG_CHECK_LAUNCH();
    void *args[] = {&g};
    SG_CHECK_CUDA(cudaLaunchCooperativeKernel(
        k.G == 4 ? (const void *)k_batched_grid<4> : (const void *)k_batched_grid<8>, grid, GB_T,
        args, smem, st));
    return SG_OK;
  }
  const int per_sm = k.threads >= 1024 ? 2 : (k.threads >= 512 ? 4 : 8);
  int grid = c->num_sms * per_sm;
  if (grid > a.nsys) grid = a.nsys;
  if (grid < 1) grid = 1;
  SG_CHECK_CUDA(cudaMemsetAsync(a.queue, 0, sizeof(int), st));
  if (k.G == 4) k_batched_pcg<4><<<grid, k.threads, 0, st>>>(a);
  else k_batched_pcg<8><<<grid, k.threads, 0, st>>>(a);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

}  // namespace
}  // namespace sg

using namespace sg;

extern "C" int sg_batched_pcg(sg_ctx *h, int32_t nsys, const int32_t *sys_ptr,
                              const int32_t *order, const sg_matrix *A, const float *b, float *x,
                              double tol, int32_t maxiters, int32_t config, int32_t *iters,
                              int32_t *status, double *relres) {
  Ctx *c = as_ctx(h);
  DeviceGuard dg_(c);
  SG_REQUIRE(c && A && sys_ptr && order && b && x && iters && status && relres,
             "sg_batched_pcg: null argument");
  SG_REQUIRE(nsys >= 1 && A->bs == 3 && A->dtype == SG_F32 && A->n >= 1,
             "sg_batched_pcg: needs >= 1 system and an FP32 3x3-blocked matrix");
  SG_REQUIRE(config >= 0 && config < kNumCfgs, "sg_batched_pcg: config %d not in [0, %d)", config,
             kNumCfgs);
  SG_REQUIRE(maxiters >= 0 && tol > 0, "sg_batched_pcg: bad tol / maxiters");
  const int64_t len = (int64_t)A->n * 3;
  Scratch s(c);
  const size_t nid = (size_t)c->num_sms * GB_MAXCTAS + nsys;  // grid-wide: segment numbers
  SG_TRY(s.reserve(Scratch::bytes_for(len, 4) * 3 + Scratch::bytes_for(A->n, sizeof(float4)) +
                   Scratch::bytes_for((size_t)A->n * 9, 4) +
                   Scratch::bytes_for(DS_N * nid, 8) + Scratch::bytes_for(DS_N * GB_W * nid, 8) +
                   Scratch::bytes_for(nid, sizeof(Seg)) + Scratch::bytes_for((size_t)nsys + 1, 4) +
                   4096));
  GridScratch w;
  BatchArgs a;
  a.nsys = nsys;
  a.sys_ptr = sys_ptr;
  a.order = order;
  a.rowptr = A->rowptr;
  a.colidx = A->colidx;
  a.vals = (const float *)A->vals;
  a.b = b;
  a.x = x;
  a.r = s.alloc<float>(len);
  w.p = s.alloc<float4>(A->n);
  a.p = (float *)w.p;  // (three floats a vertex in the per-system kernel)
  a.q = s.alloc<float>(len);
  a.z = s.alloc<float>(len);
  a.dinv = s.alloc<float>((size_t)A->n * 9);
  a.queue = s.alloc<int>(1);
  a.iters = iters;
  a.status = status;
  a.relres = relres;
  a.tol = tol;
  a.maxiters = maxiters;
  w.part = s.alloc<double>(DS_N * nid);
  w.wps = s.alloc<double>(DS_N * GB_W * nid);
  w.segs = s.alloc<Seg>(nid);
  w.chunk_ptr = s.alloc<int32_t>((size_t)nsys + 1);
  w.bar = s.alloc<unsigned int>(2);
  return launch(c, c->stream, a, config, A->n, A->nnzb, w);
}

extern "C" int sg_batched_configs(void) { return kNumCfgs; }

// Element assembly, row tiles: a CTA owns a run of consecutive block rows
// and assembles them from shared memory.
//
// The row owners of sg_assemble.cuh walk a row's incidences one after the
// other, each a chain of dependent loads, and compute an element once per
// (row, column, block row).  Here, for a tile of rows:
//
//   1. one thread per incidence (e, i) reads the element's endpoints and
//      finds the column position of each in row v (the tile's columns are in
//      shared memory); it marks the incidence in the bit mask of each of its
//      slots (bit k = the row's k-th incidence);
//   2. each distinct element of the tile (a small hash table finds them) is
//      evaluated once into a record in shared memory;
//   3. one thread per slot walks its mask in ascending bit order -- ascending
//      element, the reference's order -- and sums the blocks in registers;
//      one thread per vector component does the same over a row's
//      incidences.  Every value is written once; no floating-point atomics.
//
// The order of every sum is the row owners' (ascending element, then
// ascending local column for an element that lists a vertex twice), so an
// element whose record holds the same rounded intermediate values gives the
// same bits as they do.
//
// What bounds it: instruction issue and the latency of the phases in FP32
// (issue 47 %, shared-memory and L1 wavefronts 53 % of peak in the linear
// map at 64^3), the one FP64 pipe of each SM (16 cycles a warp instruction)
// in FP64.  At 96^3, Morton order, map by map against the kernels before
// (element blocks written out and gathered, or one group of lanes a row):
//   linear FP32 stiffness + force 3.20 -> 1.6 ms (with the element-blocks
//   plan), 7.6 -> 1.65 ms (without); neo-Hookean FP32 10.3 -> 2.1, FP64
//   60 -> 18; heat FP32 1.4 -> 0.77, FP64 10.3 -> 2.3 ms.
// At 128^3 the linear map takes 3.7 ms (was 7.6), at 64^3 the neo-Hookean
// one 0.63 (3.0).
// 32 rows a tile: 16 rows cost 2.35 ms in the linear map (3.0 evaluations an
// element instead of 2.3); 64 rows the same 1.56 ms in Morton order, but in
// lattice order, where a run of rows shares fewer elements, their records
// overflow the buffers and the tiles are taken again in parts (6.6 ms against
// 1.7).  128 threads a tile: 2 % to 30 % slower; 512: twice as slow.
#pragma once
#include "sg_assemble.cuh"

namespace sg {

constexpr int TILE_T = 256;
constexpr int TILE_MAXROWS = 32;
constexpr int TILE_Q = 3;  // incidences in flight a thread

struct TileCfg {
  int rows;                    // rows per CTA
  int icap, scap, mcap, ucap;  // incidences, slots, mask words, element records
  int hcap;                    // element table entries, a power of two > ucap
  int maxrow;                  // longest row the mesh declares
  int pre;                     // an element's terms are summed before they join a slot
  int step;                    // largest power of two <= longest row's bound
  int ep16;                    // endpoints (and slots) can be read 16 bytes at a time
  const uint32_t *slots;       // element-to-slot map, or null: columns are searched
};

// ---------------------------------------------------------------------------
// Elements.  Each provides
//   CARD, BS, HAS_MAT, HAS_VEC
//   NREC (values of an element's record, a stride that spreads random
//   records over the banks)
//   stage(a, e, vv, rec): evaluate the element (endpoints vv)
//   on(a, v, u): whether slot (v, u) takes the element terms (constraints)
//   add(rec, i, j, on, pre, acc): acc += block (i, j), term by term or (pre)
//     the terms summed first
//   vec(rec, i, l, acc): acc += component l of vertex i's term
//   fin_block / fin_vec as in sg_assemble.cuh
// ---------------------------------------------------------------------------
__device__ __forceinline__ void ld_vec4(const float *p, float v[4]) {
  const float4 t = *reinterpret_cast<const float4 *>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void ld_vec4(const double *p, double v[4]) {
  v[0] = p[0]; v[1] = p[1]; v[2] = p[2]; v[3] = p[3];
}

// Values per staged 3-vector: padded to one 16-byte load in FP32.
template <typename T> struct tile_vec { static constexpr int S = sizeof(T) == 4 ? 4 : 3; };
__device__ __forceinline__ void ld_vec3(const float *p, float v[3]) {
  const float4 t = *reinterpret_cast<const float4 *>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z;
}
__device__ __forceinline__ void ld_vec3(const double *p, double v[3]) {
  v[0] = p[0]; v[1] = p[1]; v[2] = p[2];
}

template <typename T> struct TileFin {
  __device__ static T fin_block(const AsmArgs<T> &, int32_t, bool, int, int, T acc) { return acc; }
  __device__ static T fin_vec(const AsmArgs<T> &, int32_t, int, T acc) { return acc; }
  __device__ static bool on(const AsmArgs<T> &, int32_t, uint32_t) { return true; }
};

// Linear tetrahedron: the closed form
//   K_ij[a][b] = h^2 W (lam g_ia g_jb + mu g_ib g_ja + mu (g_i . g_j) dab),
// algebraically fem_linear.sim's W Bm' E Bm.  Every product pairs a factor
// of each vertex and nothing is contracted, so the (j, i) block is bitwise
// the transpose of (i, j) and, summed in the same element order, the matrix
// is exactly symmetric (the symmetric-storage SpMV reads only its upper
// half).
template <typename T> struct LinTetTile : TileFin<T> {
  static constexpr int CARD = 4, BS = 3;
  static constexpr bool HAS_MAT = true, HAS_VEC = false;
  // four gradients, then lam, mu, h^2 W, mass
  static constexpr int VS = tile_vec<T>::S, NREC = sizeof(T) == 4 ? 20 : 17;
  __device__ static bool on(const AsmArgs<T> &a, int32_t v, uint32_t u) {
    return a.c[v] <= 0 && a.c[u] <= 0;
  }
  __device__ static void stage(const AsmArgs<T> &a, int64_t e, const int32_t *vv, T *rec) {
    T *co = rec + 4 * VS;
    const T *Bt = a.B + 9 * e;
    T b[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) b[q] = Bt[q];
    const T W = a.W[e];
    co[0] = a.lam[e];
    co[1] = a.mu[e];
    co[2] = mul_rn(mul_rn(a.h, a.h), W);
    co[3] = (T(0.25) * a.rho) * W;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      rec[d] = b[d];
      rec[VS + d] = b[3 + d];
      rec[2 * VS + d] = b[6 + d];
      rec[3 * VS + d] = ((T(0) - b[d]) - b[3 + d]) - b[6 + d];
    }
  }
  __device__ static void add(const T *rec, int i, int j, bool on, bool pre, T *acc) {
    T k[4], gi[3], gj[3];
    ld_vec4(rec + 4 * VS, k);
    if (on) {
      ld_vec3(rec + i * VS, gi);
      ld_vec3(rec + j * VS, gj);
      const T lm = k[0], u = k[1], hw = k[2];
      const T ug =
          mul_rn(u, add_rn(add_rn(mul_rn(gi[0], gj[0]), mul_rn(gi[1], gj[1])),
                           mul_rn(gi[2], gj[2])));
#pragma unroll
      for (int l = 0; l < 3; ++l)
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          T t = add_rn(mul_rn(lm, mul_rn(gi[l], gj[m])), mul_rn(u, mul_rn(gi[m], gj[l])));
          if (l == m) t = add_rn(t, ug);
          t = mul_rn(hw, t);
          if (l == m && pre && i == j) t = add_rn(t, k[3]);
          acc[l * 3 + m] = add_rn(acc[l * 3 + m], t);
        }
    }
    if (i == j && !(pre && on)) {
#pragma unroll
      for (int l = 0; l < 3; ++l) acc[l * 4] += k[3];
    }
  }
  __device__ static void vec(const T *, int, int, T &) {}
};

// Neo-Hookean tangent (femTet.sim compute_stiffness) in closed form: with
// q_i = F^-T g_i, block (i, j) is
//   h^2 W [ mu (g_i . g_j) I + (mu - lam log J) q_j q_i' + lam q_i q_j' ],
// which is the twelve dPdF products of the program contracted by hand.
template <typename T> struct NeoTile : TileFin<T> {
  static constexpr int CARD = 4, BS = 3;
  static constexpr bool HAS_MAT = true, HAS_VEC = false;
  // four q, then mu (g_i . g_j), two moduli, mass
  static constexpr int VS = tile_vec<T>::S, NREC = sizeof(T) == 4 ? 36 : 25;
  __device__ static bool on(const AsmArgs<T> &a, int32_t v, uint32_t u) {
    return a.c[v] <= 0 && a.c[u] <= 0;
  }
  __device__ static void stage(const AsmArgs<T> &a, int64_t e, const int32_t *vv, T *rec) {
    T *co = rec + 4 * VS;
    T F[9], Fi[9], g[4][3];
    const T *Bt = a.B + 9 * e;
    tet_F(a, e, F);
    const T u = a.mu[e], l = a.lam[e], W = a.W[e];
    const T JJ = d_log(d_det3(F));
    d_inv3(F, Fi);
    const T hw = (a.h * a.h) * W, hu = hw * u;
    co[10] = hw * (u - l * JJ);
    co[11] = hw * l;
    co[12] = (T(0.25) * a.rho) * W;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      g[0][d] = Bt[d]; g[1][d] = Bt[3 + d]; g[2][d] = Bt[6 + d];
      g[3][d] = -((Bt[d] + Bt[3 + d]) + Bt[6 + d]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int d = 0; d < 3; ++d)
        rec[i * VS + d] = (Fi[d] * g[i][0] + Fi[3 + d] * g[i][1]) + Fi[6 + d] * g[i][2];
    int k = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = i; j < 4; ++j)
        co[k++] = hu * ((g[i][0] * g[j][0] + g[i][1] * g[j][1]) + g[i][2] * g[j][2]);
  }
  __device__ static void add(const T *rec, int i, int j, bool on, bool pre, T *acc) {
    const T *co = rec + 4 * VS;
    if (on) {
      T qi[3], qj[3];
      ld_vec3(rec + i * VS, qi);
      ld_vec3(rec + j * VS, qj);
      const int lo = min(i, j), hi = max(i, j);
      const T ug = co[tri_index(4, lo, hi)], hc = co[10], hl = co[11];
#pragma unroll
      for (int l = 0; l < 3; ++l)
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          acc[l * 3 + m] += hc * (qj[l] * qi[m]);
          acc[l * 3 + m] += hl * (qi[l] * qj[m]);
          if (l == m) acc[l * 3 + m] += ug;
        }
    }
    if (i == j) {
#pragma unroll
      for (int l = 0; l < 3; ++l) acc[l * 4] += co[12];
    }
  }
  __device__ static void vec(const T *, int, int, T &) {}
};

// P1 heat: the ten distinct values of the element matrix and the four of its
// vector, once per element, so that a slot's sum is one addition a block (the
// FP64 pipe bounds the FP64 map).  EXACT: the reference's operations in its
// order; else contracted, with the vector from the sum of T0.  The fourth
// gradient is formed before it is multiplied: products with it taken from the
// other three vertices' (g_3 . g_3 = sum of g_i . g_j) lose the square of a
// slender element's aspect ratio instead of the ratio itself, in FP32 the sign
// of the diagonal at 1,000.  (At 96^3 that saves FP64 2.28 -> 2.10 ms, FP32
// nothing: 0.77.)
template <typename T, bool EXACT> struct HeatTile : TileFin<T> {
  static constexpr int CARD = 4, BS = 1;
  static constexpr bool HAS_MAT = true, HAS_VEC = true;
  static constexpr int NREC = 15;
  __device__ static void stage(const AsmArgs<T> &a, int64_t e, const int32_t *vv, T *rec) {
    T g[4][3], t[4];
#pragma unroll
    for (int q = 0; q < 9; ++q) g[q / 3][q % 3] = a.B[9 * e + q];
#pragma unroll
    for (int d = 0; d < 3; ++d) g[3][d] = -((g[0][d] + g[1][d]) + g[2][d]);
#pragma unroll
    for (int j = 0; j < 4; ++j) t[j] = a.T0[vv[j]];
    const T W = a.W[e], kw = (a.dt * a.kappa[e]) * W;
    if (EXACT) {
      const T mw = W / T(20.0), mw2 = T(2.0) * mw;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        T bi = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const T mij = i == j ? mw2 : mw;
          bi += mij * t[j];
          if (j >= i)
            rec[tri_index(4, i, j)] =
                mij + kw * ((g[i][0] * g[j][0] + g[i][1] * g[j][1]) + g[i][2] * g[j][2]);
        }
        rec[10 + i] = bi;
      }
    } else {
      const T mw = W * T(0.05), mw2 = T(2.0) * mw;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = i; j < 4; ++j)
          rec[tri_index(4, i, j)] =
              (i == j ? mw2 : mw) +
              kw * ((g[i][0] * g[j][0] + g[i][1] * g[j][1]) + g[i][2] * g[j][2]);
      const T ts = (t[0] + t[1]) + (t[2] + t[3]);
#pragma unroll
      for (int i = 0; i < 4; ++i) rec[10 + i] = mw * (ts + t[i]);
    }
  }
  __device__ static void add(const T *rec, int i, int j, bool on, bool pre, T *acc) {
    acc[0] += rec[tri_index(4, min(i, j), max(i, j))];
  }
  __device__ static void vec(const T *rec, int i, int, T &acc) {
    acc += rec[10 + i];
  }
};

// compute_force of femTet.sim / fem_linear.sim: each vertex's terms (elastic,
// then gravity and velocity) summed once per element.
template <typename T, bool NEO> struct TetForceTile : TileFin<T> {
  static constexpr int CARD = 4, BS = 3;
  static constexpr bool HAS_MAT = false, HAS_VEC = true;
  static constexpr int NREC = 13;
  __device__ static void stage(const AsmArgs<T> &a, int64_t e, const int32_t *vv, T *rec) {
    const T u = a.mu[e], lm = a.lam[e], W = a.W[e];
    T F[9], P[9], H[9];
    tet_F(a, e, F);
    if (NEO) {
      const T JJ = d_log(d_det3(F));
      T Fi[9], FinvT[9];
      d_inv3(F, Fi);
      d_tr3(Fi, FinvT);
#pragma unroll
      for (int q = 0; q < 9; ++q) P[q] = (u * (F[q] - FinvT[q])) + ((lm * JJ) * FinvT[q]);
    } else {
      T FI[9];
#pragma unroll
      for (int q = 0; q < 9; ++q) FI[q] = F[q] - T((q % 4) == 0);
      const T tr = (FI[0] + FI[4]) + FI[8];
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int s2 = 0; s2 < 3; ++s2)
          P[r * 3 + s2] = (u * (FI[r * 3 + s2] + FI[s2 * 3 + r])) + ((lm * tr) * T(r == s2));
    }
    tet_H(W, P, a.B + 9 * e, H);
    const T m = (T(0.25) * a.rho) * W;
#pragma unroll
    for (int l = 0; l < 3; ++l) {
      const T fg = m * a.grav[l];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        T t = i < 3 ? a.h * H[l * 3 + i] : (-a.h) * H[l * 3];
        if (i == 3) {
          t += (-a.h) * H[l * 3 + 1];
          t += (-a.h) * H[l * 3 + 2];
        }
        t += (a.h * fg) + (m * a.v[(int64_t)vv[i] * 3 + l]);
        rec[i * 3 + l] = t;
      }
    }
  }
  __device__ static void add(const T *, int, int, bool, bool, T *) {}
  __device__ static void vec(const T *rec, int i, int l, T &acc) {
    acc += rec[i * 3 + l];
  }
  __device__ static T fin_vec(const AsmArgs<T> &a, int32_t v, int, T acc) {
    return a.c[v] > 0 ? T(0) : acc;  // nothing to a constrained vertex
  }
};

// Springs: the 3x3 k and the force of SpringElem, once per spring.
template <typename T> struct SpringTile {
  static constexpr int CARD = 2, BS = 3;
  static constexpr bool HAS_MAT = true, HAS_VEC = true;
  static constexpr int NREC = 13;
  // a spring between free points writes all four blocks, else only the free
  // end's diagonal one
  __device__ static bool on(const AsmArgs<T> &a, int32_t v, uint32_t u) {
    return !a.fixed[v] && !a.fixed[u];
  }
  __device__ static void stage(const AsmArgs<T> &a, int64_t e, const int32_t *vv, T *rec) {
#pragma unroll
    for (int l = 0; l < 3; ++l) SpringElem<T>::kfe(a, e, l, rec + 3 * l, rec[9 + l]);
  }
  __device__ static void add(const T *rec, int i, int j, bool on, bool pre, T *acc) {
    if (!on) return;
#pragma unroll
    for (int q = 0; q < 9; ++q) acc[q] += (i != j) ? -rec[q] : rec[q];
  }
  __device__ static void vec(const T *rec, int i, int l, T &acc) {
    acc += (i == 0) ? rec[9 + l] : -rec[9 + l];
  }
  __device__ static T fin_block(const AsmArgs<T> &a, int32_t v, bool dg, int l, int m, T acc) {
    return SpringElem<T>::fin_block(a, v, dg, l, m, acc);
  }
  __device__ static T fin_vec(const AsmArgs<T> &a, int32_t v, int l, T acc) {
    return SpringElem<T>::fin_vec(a, v, l, a.fixed[v] ? T(0) : acc);
  }
};

// Scalar springs of cg.sim (ScalarSpringElem).
template <typename T> struct ScalarSpringTile {
  static constexpr int CARD = 2, BS = 1;
  static constexpr bool HAS_MAT = true, HAS_VEC = false;
  static constexpr int NREC = 1;
  __device__ static void stage(const AsmArgs<T> &a, int64_t e, const int32_t *vv, T *rec) {
    rec[0] = a.a[e];
  }
  __device__ static void add(const T *rec, int i, int j, bool on, bool pre, T *acc) {
    acc[0] += (i == j) ? rec[0] : -rec[0];
  }
  __device__ static void vec(const T *, int, int, T &) {}
  __device__ static T fin_block(const AsmArgs<T> &a, int32_t v, bool dg, int l, int m, T acc) {
    return ScalarSpringElem<T>::fin_block(a, v, dg, l, m, acc);
  }
  __device__ static T fin_vec(const AsmArgs<T> &, int32_t, int, T acc) { return acc; }
  __device__ static bool on(const AsmArgs<T> &, int32_t, uint32_t) { return true; }
};

// ---------------------------------------------------------------------------
// Kernel
// ---------------------------------------------------------------------------
// Bytes of the element table and list; step 3 stages its output in the same
// place.
template <class E, typename T> __host__ __device__ inline size_t tile_table(const TileCfg &g) {
  size_t b = (size_t)g.ucap * 4 + (size_t)g.hcap * 6;
  const size_t out = E::HAS_MAT && E::BS > 1 ? (size_t)TILE_T * E::BS * E::BS * sizeof(T) : 0;
  if (b < out) b = out;
  return (b + 15) & ~size_t(15);
}
template <class E, typename T> __host__ __device__ inline size_t tile_smem(const TileCfg &g) {
  size_t b = ((size_t)g.ucap * E::NREC * sizeof(T) + 15) & ~size_t(15);
  b += tile_table<E, T>(g) + (size_t)g.icap * 4;  // info
  if (E::HAS_MAT) b += (size_t)g.icap * 4 + (size_t)g.scap * 5 + (size_t)g.mcap * 4;
  return (b + 15) & ~size_t(15);
}

template <int CARD>
__device__ __forceinline__ void tile_endpoints(const int32_t *ep, int64_t e, int ep16,
                                               int32_t *vv) {
  if (CARD == 4 && ep16) {
    const int4 t = reinterpret_cast<const int4 *>(ep)[e];
    vv[0] = t.x; vv[1 % CARD] = t.y; vv[2 % CARD] = t.z; vv[3 % CARD] = t.w;
  } else {
#pragma unroll
    for (int j = 0; j < CARD; ++j) vv[j] = ep[e * CARD + j];
  }
}

// A row too large for the tile's buffers: every thread takes slots (and
// vector components) of the row and evaluates each of its elements itself,
// in the same order.
template <class E, typename T>
__device__ __noinline__ void tile_big_row(const AsmArgs<T> &a, int32_t v, const TileCfg &g) {
  constexpr int CARD = E::CARD, BS = E::BS;
  const uint32_t i0 = a.ve_ptr[v], i1 = a.ve_ptr[v + 1];
  uint32_t r0 = 0, len = 0;
  if (E::HAS_MAT) {
    r0 = a.rowptr[v];
    len = a.rowptr[v + 1] - r0;
    if ((int64_t)len > g.maxrow) {
      if (threadIdx.x == 0) atomicCAS(a.err, 0, 4 /* DEV_ROW_OVERFLOW */);
      return;
    }
  }
  const uint32_t nvec = E::HAS_VEC ? BS : 0;
  for (uint32_t t = threadIdx.x; t < len + nvec; t += blockDim.x) {
    T acc[BS * BS];
#pragma unroll
    for (int q = 0; q < BS * BS; ++q) acc[q] = T(0);
    T va = T(0);
    const uint32_t col = t < len ? a.colidx[r0 + t] : 0u;
    const bool on = t < len && E::on(a, v, col);
    for (uint32_t k = i0; k < i1; ++k) {
      const uint32_t id = a.ve_idx[k];
      const int64_t e = id / (uint32_t)CARD;
      const int i = (int)(id % (uint32_t)CARD);
      int32_t vv[CARD];
      bool used = t >= len;
#pragma unroll
      for (int j = 0; j < CARD; ++j) {
        vv[j] = a.ep[e * CARD + j];
        used = used || (uint32_t)vv[j] == col;
      }
      if (!used) continue;
      __align__(16) T rec[E::NREC];
      E::stage(a, e, vv, rec);
      if (t >= len) {
        E::vec(rec, i, (int)(t - len), va);
      } else {
        for (int j = 0; j < CARD; ++j)
          if ((uint32_t)vv[j] == col) E::add(rec, i, j, on, g.pre, acc);
      }
    }
    if (t >= len) {
      a.f[(int64_t)v * BS + (t - len)] = E::fin_vec(a, v, (int)(t - len), va);
    } else {
#pragma unroll
      for (int q = 0; q < BS * BS; ++q)
        a.vals[(size_t)(r0 + t) * BS * BS + q] =
            E::fin_block(a, v, col == (uint32_t)v, q / BS, q % BS, acc[q]);
    }
  }
}

template <class E, typename T>
__global__ void __launch_bounds__(TILE_T, 3) k_tile(AsmArgs<T> a, TileCfg g) {
  constexpr int CARD = E::CARD, BS = E::BS, NB = BS * BS;
  extern __shared__ __align__(16) unsigned char tile_raw[];
  __shared__ uint32_t ip[TILE_MAXROWS + 1], sp[TILE_MAXROWS + 1], mp[TILE_MAXROWS + 1];
  __shared__ int dpos[TILE_MAXROWS];
  __shared__ int nrec, nitem;
  unsigned char *raw = tile_raw;
  T *rec = reinterpret_cast<T *>(raw);
  raw += ((size_t)g.ucap * E::NREC * sizeof(T) + 15) & ~size_t(15);
  T *out = reinterpret_cast<T *>(raw);
  uint32_t *elem = reinterpret_cast<uint32_t *>(raw);    // element of each record
  uint32_t *hkey = elem + g.ucap;                        // element table: element, record
  uint16_t *hval = reinterpret_cast<uint16_t *>(hkey + g.hcap);
  raw += tile_table<E, T>(g);
  uint32_t *info = reinterpret_cast<uint32_t *>(raw);    // record | i << 16
  uint32_t *spos = info + g.icap;                        // four 8-bit column positions
  uint32_t *cols = spos + (E::HAS_MAT ? g.icap : 0);
  uint32_t *mask = cols + (E::HAS_MAT ? g.scap : 0);
  uint8_t *srow = reinterpret_cast<uint8_t *>(mask + (E::HAS_MAT ? g.mcap : 0));

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int32_t v0 = blockIdx.x * g.rows;
  const int nr = min(g.rows, a.n - v0);
  for (int r = tid; r <= nr; r += TILE_T) {
    ip[r] = a.ve_ptr[v0 + r];
    if (E::HAS_MAT) sp[r] = a.rowptr[v0 + r];
  }
  __syncthreads();
  if (E::HAS_MAT) {
    // prefix sum of the rows' mask words; a row that 8-bit positions cannot
    // address or that is longer than declared counts as too large
    if (warp == 0) {
      uint32_t w = 0;
      if (lane < nr) {
        const uint32_t len = sp[lane + 1] - sp[lane], wr = (ip[lane + 1] - ip[lane] + 31) / 32;
        w = len > 254 || (int)len > g.maxrow || wr > 1024 ? (1u << 24) : len * wr;
      }
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += t;
      }
      mp[lane + 1] = w;
      if (lane == 0) mp[0] = 0;
    }
    __syncthreads();
  }
  int limit = nr;
  for (int rb = 0; rb < nr;) {
    // the rows of this pass: as many as the buffers hold
    bool ok = false;
    if (tid < nr - rb && tid < limit) {
      const int e1 = rb + tid + 1;
      ok = ip[e1] - ip[rb] <= (uint32_t)g.icap;
      if (E::HAS_MAT)
        ok = ok && sp[e1] - sp[rb] <= (uint32_t)g.scap && mp[e1] - mp[rb] <= (uint32_t)g.mcap;
    }
    const int fit = __syncthreads_count(ok);
    if (fit == 0) {
      tile_big_row<E, T>(a, v0 + rb, g);
      ++rb;
      continue;
    }
    const int re = rb + fit;
    const uint32_t I0 = ip[rb];
    const int I = (int)(ip[re] - I0);
    const uint32_t S0 = E::HAS_MAT ? sp[rb] : 0u, M0 = E::HAS_MAT ? mp[rb] : 0u;
    const int S = E::HAS_MAT ? (int)(sp[re] - S0) : 0;
    if (tid == 0) nrec = nitem = 0;
    // the first TILE_Q incidences a thread, in flight while the tables clear
    uint32_t ids[TILE_Q];
#pragma unroll
    for (int q = 0; q < TILE_Q; ++q)
      ids[q] = q * TILE_T + tid < I ? a.ve_idx[I0 + q * TILE_T + tid] : 0u;
    for (int h = tid; h < g.hcap; h += TILE_T) hkey[h] = 0xffffffffu;
    if (E::HAS_MAT) {
      const int M = (int)(mp[re] - M0);
      for (int m = tid; m < M; m += TILE_T) mask[m] = 0u;
#pragma unroll 4
      for (int s = tid; s < S; s += TILE_T) cols[s] = a.colidx[S0 + s];
      if (tid < TILE_MAXROWS) dpos[tid] = -1;
      for (int r = rb + warp; r < re; r += TILE_T / 32)
        for (uint32_t s = sp[r] - S0 + lane; s < sp[r + 1] - S0; s += 32) srow[s] = (uint8_t)r;
    }
    __syncthreads();
    // 1. incidences, TILE_Q a thread at a time: their endpoints (or slots)
    // are all in flight before the first is used
    for (int k0 = 0; k0 < I; k0 += TILE_T * TILE_Q) {
      if (k0) {
#pragma unroll
        for (int q = 0; q < TILE_Q; ++q) {
          const int k = k0 + q * TILE_T + tid;
          ids[q] = k < I ? a.ve_idx[I0 + k] : 0u;
        }
      }
      uint32_t four[TILE_Q][CARD];  // endpoints, or slots
      if (E::HAS_MAT) {
#pragma unroll
        for (int q = 0; q < TILE_Q; ++q) {
          if (g.slots) {
            if (CARD == 4 && g.ep16) {
              const uint4 t = reinterpret_cast<const uint4 *>(g.slots)[ids[q]];
              four[q][0] = t.x; four[q][1 % CARD] = t.y;
              four[q][2 % CARD] = t.z; four[q][3 % CARD] = t.w;
            } else {
#pragma unroll
              for (int j = 0; j < CARD; ++j) four[q][j] = g.slots[(size_t)ids[q] * CARD + j];
            }
          } else {
            int32_t vv[CARD];
            tile_endpoints<CARD>(a.ep, ids[q] / (uint32_t)CARD, g.ep16, vv);
#pragma unroll
            for (int j = 0; j < CARD; ++j) four[q][j] = (uint32_t)vv[j];
          }
        }
      }
#pragma unroll
      for (int q = 0; q < TILE_Q; ++q) {
      const int k = k0 + q * TILE_T + tid;
      if (k0 + q * TILE_T >= I) break;
      bool own = false;
      uint32_t e = 0, h = 0;
      if (k < I) {
        const uint32_t id = ids[q];
        e = id / (uint32_t)CARD;
        const int i = (int)(id - e * (uint32_t)CARD);
        if (E::HAS_MAT) {
          uint32_t pos4 = 0xffffffffu;
          int r;
          uint32_t len, lo[CARD];
          if (g.slots) {
            const uint32_t s0 = four[q][0] - S0;
            r = s0 < (uint32_t)S ? (int)srow[s0] : rb;
            len = sp[r + 1] - sp[r];
#pragma unroll
            for (int j = 0; j < CARD; ++j) lo[j] = four[q][j] - sp[r];
          } else {
            uint32_t vi = four[q][0];
#pragma unroll
            for (int j = 1; j < CARD; ++j) vi = i == j ? four[q][j] : vi;
            r = (int)vi - v0;
            const uint32_t c0 = sp[r] - S0;
            len = sp[r + 1] - sp[r];
            // the columns below each endpoint, all endpoints a step at a time
#pragma unroll
            for (int j = 0; j < CARD; ++j) lo[j] = 0;
            for (uint32_t st = g.step; st; st >>= 1) {
#pragma unroll
              for (int j = 0; j < CARD; ++j) {
                const uint32_t t = lo[j] + st;
                if (t <= len && cols[c0 + t - 1] < four[q][j]) lo[j] = t;
              }
            }
#pragma unroll
            for (int j = 0; j < CARD; ++j)
              if (lo[j] < len && cols[c0 + lo[j]] != four[q][j]) lo[j] = len;
          }
          const uint32_t wr = (ip[r + 1] - ip[r] + 31) / 32, kr = (uint32_t)k - (ip[r] - I0);
          uint32_t *mrow = mask + (mp[r] - M0) + (kr >> 5);
#pragma unroll
          for (int j = 0; j < CARD; ++j) {
            if (lo[j] >= len || (kr >> 5) >= wr) {
              atomicCAS(a.err, 0, 3 /* DEV_SLOT_MISSING */);
              continue;
            }
            pos4 = (pos4 & ~(0xffu << (8 * j))) | (lo[j] << (8 * j));
            atomicOr(&mrow[lo[j] * wr], 1u << (kr & 31));
          }
          spos[k] = pos4;
        }
        // the element's table entry; the thread that makes it owns the record
        h = (e * 0x9E3779B1u) >> 16;
        int probe = 0;
        for (;; ++h, ++probe) {
          h &= (uint32_t)g.hcap - 1u;
          const uint32_t old = atomicCAS(&hkey[h], 0xffffffffu, e);
          own = old == 0xffffffffu;
          if (own || old == e || probe >= g.hcap) break;
        }
        if (probe >= g.hcap) atomicMax(&nrec, 2 * g.hcap);  // full: more elements than records
        info[k] = h | ((uint32_t)i << 16);
      }
      const unsigned b = __ballot_sync(0xffffffffu, own);
      int base = 0;
      if (lane == 0 && b) base = atomicAdd(&nrec, __popc(b));
      base = __shfl_sync(0xffffffffu, base, 0) + __popc(b & ((1u << lane) - 1u));
      if (own && base < g.ucap) {
        elem[base] = e;
        hval[h] = (uint16_t)base;
      }
      }
    }
    __syncthreads();
    const int U = nrec;
    if (U > g.ucap) {  // more distinct elements than records: fewer rows, from here on
      __syncthreads();
      if (fit == 1) {
        tile_big_row<E, T>(a, v0 + rb, g);
        ++rb;
      } else {
        limit = max(1, min(fit - 1, (int)((int64_t)fit * g.ucap * 7 / ((int64_t)U * 8))));
      }
      continue;
    }
    // 2. the incidences' records, and the elements' values in them
    for (int k = tid; k < I; k += TILE_T) {
      const uint32_t w = info[k];
      info[k] = (w & 0xffff0000u) | hval[w & 0xffffu];
    }
    if (E::HAS_MAT)
      for (int s = tid; s < S; s += TILE_T) {
        const int r = srow[s];
        if (cols[s] == (uint32_t)(v0 + r)) dpos[r] = s;
      }
    int32_t vv[CARD], nx[CARD];
    if (tid < U) tile_endpoints<CARD>(a.ep, elem[tid], g.ep16, nx);
    for (int u = tid; u < U; u += TILE_T) {
#pragma unroll
      for (int j = 0; j < CARD; ++j) vv[j] = nx[j];
      if (u + TILE_T < U) tile_endpoints<CARD>(a.ep, elem[u + TILE_T], g.ep16, nx);
      E::stage(a, elem[u], vv, rec + (size_t)u * E::NREC);
    }
    __syncthreads();
    // 3. sums, a warp an item: 32 diagonal slots (a row's longest, first), 32
    // vector components, then 32 consecutive slots without the diagonal ones
    const int rows = re - rb;
    const int nd = E::HAS_MAT ? (rows + 31) / 32 : 0;
    const int nv = E::HAS_VEC ? (rows * BS + 31) / 32 : 0;
    const int items = nd + nv + (S + 31) / 32;
    for (;;) {
      int it = 0;
      if (lane == 0) it = atomicAdd(&nitem, 1);
      it = __shfl_sync(0xffffffffu, it, 0);
      if (it >= items) break;
      if (E::HAS_VEC && it >= nd && it < nd + nv) {
        const int t = (it - nd) * 32 + lane;
        if (t < rows * BS) {
          const int r = rb + t / BS, l = t % BS;
          T va = T(0);
          const int k1 = (int)(ip[r + 1] - I0);
          for (int k = (int)(ip[r] - I0); k < k1; ++k) {
            const uint32_t w = info[k];
            E::vec(rec + (w & 0xffffu) * E::NREC, (int)(w >> 16), l, va);
          }
          a.f[(int64_t)(v0 + r) * BS + l] = E::fin_vec(a, v0 + r, l, va);
        }
        continue;
      }
      if (!E::HAS_MAT) continue;
      const bool dgi = it < nd;
      const int s0 = (it - nd - nv) * 32;
      int s = dgi ? S : s0 + lane, r = 0;
      if (dgi) {
        r = rb + it * 32 + lane;
        if (r < re && dpos[r] >= 0) s = dpos[r];
      } else if (s < S) {
        r = srow[s];
        if (cols[s] == (uint32_t)(v0 + r)) s = S;
      }
      const bool act = s < S;
      T acc[NB];
#pragma unroll
      for (int q = 0; q < NB; ++q) acc[q] = T(0);
      if (act) {
        const uint32_t pos = (uint32_t)s - (sp[r] - S0), rep = pos * 0x01010101u;
        const int kr = (int)(ip[r] - I0), wr = (int)((ip[r + 1] - ip[r] + 31) / 32);
        const uint32_t *m = mask + (mp[r] - M0) + pos * wr;
        const bool on = E::on(a, v0 + r, cols[s]);
        for (int w = 0; w < wr; ++w) {
          uint32_t bits = m[w];
          while (bits) {
            const int k = kr + w * 32 + __ffs(bits) - 1;
            bits &= bits - 1u;
            const uint32_t inf = info[k], x = spos[k] ^ rep;
            // bit 7 of each byte of x that is zero: the endpoints in this column
            uint32_t eq = ~(((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x | 0x7f7f7f7fu);
            do {  // more than one match: the element lists the vertex twice
              const int j = (__ffs(eq) - 1) >> 3;
              eq &= eq - 1u;
              E::add(rec + (inf & 0xffffu) * E::NREC, (int)(inf >> 16), j, on, g.pre, acc);
            } while (eq);
          }
        }
#pragma unroll
        for (int q = 0; q < NB; ++q)
          acc[q] = E::fin_block(a, v0 + r, dgi, q / BS, q % BS, acc[q]);
      }
      if (BS == 1 || dgi) {
        if (act) {
#pragma unroll
          for (int q = 0; q < NB; ++q) a.vals[(size_t)(S0 + s) * NB + q] = acc[q];
        }
      } else {
        // through shared memory to lane-consecutive stores
        T *st = out + warp * 32 * NB;
#pragma unroll
        for (int q = 0; q < NB; ++q) st[lane * NB + q] = acc[q];
        const unsigned on = __ballot_sync(0xffffffffu, act);
        __syncwarp();
        T *dst = a.vals + (size_t)(S0 + s0) * NB;
#pragma unroll
        for (int q = 0; q < NB; ++q) {
          const int x = lane + 32 * q;
          if ((on >> (x / NB)) & 1u) dst[x] = st[x];
        }
        __syncwarp();
      }
    }
    __syncthreads();
    rb = re;
  }
}

}  // namespace sg

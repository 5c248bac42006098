// Host launchers of the assembly kernels.  Included by sg_assemble_exact.cu
// (compiled with --fmad=false, namespace sg::exact) and sg_assemble_fast.cu
// (default contraction, namespace sg::fast); SG_ASM_NS names the namespace
// and SG_ASM_EXACT selects the operation-order-exact element forms.
#include "sg_assemble.cuh"
#include "sg_assemble_tile.cuh"
#include "sg_internal.cuh"
#include "sg_asm_api.h"

namespace sg {
namespace SG_ASM_NS {

template <class Elem, int G, int BS, typename T>
static int launch_rows(Ctx *c, AsmArgs<T> &a) {
  if (a.n == 0) return SG_OK;
  const int maxrow = Elem::HAS_MAT ? a.maxrow : 0;
  const size_t per_group = (size_t)maxrow * (BS * BS * sizeof(T) + 4);
  int threads = 128;
  while (threads > G && (threads / G) * per_group > 96 * 1024) threads >>= 1;
  if ((threads / G) * per_group > 96 * 1024)
    return set_error(SG_ERR_UNSUPPORTED, "assembly: a row of %d blocks exceeds shared memory",
                     maxrow);
  const size_t sh = (threads / G) * per_group;
  if (sh > 48 * 1024)
    SG_CHECK_CUDA(cudaFuncSetAttribute(k_rows<Elem, G, BS, T>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh));
  a.err = c->d_err;
  const int grid = grid_for(c, (int64_t)a.n * G, threads, 16);
  k_rows<Elem, G, BS, T><<<grid, threads, sh, c->stream>>>(a);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

// Row tiles (sg_assemble_tile.cuh).  Rows a tile: 32, halved while the tiles
// are fewer than two an SM or their buffers exceed half of an SM's shared
// memory.  The buffers hold 15 % more than the mesh's average, and a record
// for three in four incidences (0.51 of them are distinct elements on a
// Morton-ordered five-tet lattice, 0.65 in lattice order); a tile that needs
// more is taken in parts.
template <class E, typename T>
static int launch_tile(Ctx *c, AsmArgs<T> &a, const sg_mesh *m) {
  if (a.n == 0) return SG_OK;
  const bool plan = m->slots && ((m->slot_src_ptr && m->slot_src) ||
                                 (m->color_order && m->color_ptr && m->ncolors > 0));
  TileCfg g;
  g.maxrow = plan ? INT32_MAX : a.maxrow;
  if (E::HAS_MAT && !plan && (size_t)a.maxrow * (E::BS * E::BS * sizeof(T) + 4) > 96 * 1024)
    return set_error(SG_ERR_UNSUPPORTED, "assembly: a row of %d blocks exceeds shared memory",
                     a.maxrow);
  // with the slot lists a block's mass joins its stiffness before the slot's
  // sum, as the caller-evaluated blocks of that plan come summed
  g.pre = m->slots && m->slot_src_ptr && m->slot_src;
  g.slots = m->slots;
  g.ep16 = (uintptr_t)a.ep % 16 == 0 && (uintptr_t)m->slots % 16 == 0;
  for (g.step = 1; g.step * 2 <= (plan ? 254 : a.maxrow) && g.step < 128;) g.step *= 2;
  const double inc = (double)a.nE * E::CARD / a.n, len = (double)a.nnzb / a.n;
  size_t sh = 0;
  for (g.rows = TILE_MAXROWS;; g.rows >>= 1) {
    g.icap = (int)(g.rows * inc * 1.15) + 32;
    if (g.icap > 32768) g.icap = 32768;
    g.ucap = (int)(g.icap * (g.rows >= 32 ? 0.75 : 0.9));
    g.scap = (int)(g.rows * len * 1.15) + 32;
    if (g.scap > 32768) g.scap = 32768;
    g.mcap = g.scap * (inc > 32 ? 3 : 1) + 64;
    for (g.hcap = 64; g.hcap < g.ucap + g.ucap / 4; g.hcap *= 2) {}
    sh = tile_smem<E, T>(g);
    const bool small = a.n < (int64_t)g.rows * 2 * c->num_sms;
    if (g.rows <= 4 || (!small && sh <= 112 * 1024)) break;
  }
  if (sh > 220 * 1024) {  // a few rows already exceed an SM: the row-by-row path
    g.icap = g.ucap = g.scap = g.mcap = 64;
    g.hcap = 128;
    sh = tile_smem<E, T>(g);
  }
  static PerDeviceOnce attr;
  SG_TRY(once_per_device(attr, c->device, []() -> int {
    SG_CHECK_CUDA(cudaFuncSetAttribute(k_tile<E, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       220 * 1024));
    return SG_OK;
  }));
  a.err = c->d_err;
  k_tile<E, T><<<(a.n + g.rows - 1) / g.rows, TILE_T, sh, c->stream>>>(a, g);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

// Caller-evaluated element blocks over the mesh's plan (fast instantiation
// only; the exact one keeps the reference's element order through the row
// owners): a gather by slot, or the blocks of one colour after another into
// cleared values.  Sets *used when it ran.
template <int BS, int CARD, typename T>
static int launch_plan(Ctx *c, AsmArgs<T> &a, const sg_mesh *m, bool *used) {
  *used = false;
  if (SG_ASM_EXACT || !m->slots) return SG_OK;
  a.err = c->d_err;
  if (m->slot_src_ptr && m->slot_src) {
    if (m->nnzb > 0) {
      k_slot_gather<BS, T><<<grid_for(c, m->nnzb * BS, 256, 8), 256, 0, c->stream>>>(
          m->nnzb, m->slot_src_ptr, m->slot_src, a.eb, a.vals);
      SG_CHECK_LAUNCH();
    }
    *used = true;
    return SG_OK;
  }
  if (!m->color_order || !m->color_ptr || m->ncolors <= 0) return SG_OK;
  SG_CHECK_CUDA(cudaMemsetAsync(a.vals, 0, (size_t)m->nnzb * BS * BS * sizeof(T), c->stream));
  for (int k = 0; k < m->ncolors; ++k) {
    const int64_t b0 = m->color_ptr[k], cnt = (int64_t)m->color_ptr[k + 1] - b0;
    if (cnt <= 0) continue;
    k_colored<BlocksElem<T, BS, CARD>, CARD, BS, T>
        <<<grid_for(c, cnt * CARD * CARD, 256, 8), 256, 0, c->stream>>>(a, m->color_order + b0,
                                                                        cnt, m->slots);
    SG_CHECK_LAUNCH();
  }
  *used = true;
  return SG_OK;
}

template <typename T>
static void fill_mesh(AsmArgs<T> &a, const sg_mesh *m) {
  a.n = m->n;
  a.card = m->card;
  a.nE = m->nE;
  a.ep = m->endpoints;
  a.ve_ptr = m->ve_ptr;
  a.ve_idx = m->ve_idx;
  a.rowptr = m->rowptr;
  a.colidx = m->colidx;
  a.maxrow = m->maxrow;
  a.nnzb = m->nnzb;
}

template <typename T>
int springs(Ctx *c, const sg_mesh *m, int form, const void *x, const void *v, const void *mass,
            const uint8_t *fixed, const void *k, const void *l0, double h, double viscous,
            const double *grav, void *vals, void *f) {
  AsmArgs<T> a;
  fill_mesh(a, m);
  a.x = (const T *)x; a.v = (const T *)v; a.m = (const T *)mass; a.fixed = fixed;
  a.k = (const T *)k; a.l0 = (const T *)l0; a.h = (T)h; a.viscous = (T)viscous;
  for (int q = 0; q < 3; ++q) a.grav[q] = (T)grav[q];
  a.form = form;
  a.vals = (T *)vals; a.f = (T *)f;
  return launch_tile<SpringTile<T>, T>(c, a, m);
}

template <typename T>
int scalar_springs(Ctx *c, const sg_mesh *m, const void *av, double diag, double scale,
                   void *vals) {
  AsmArgs<T> a;
  fill_mesh(a, m);
  a.a = (const T *)av; a.diag = (T)diag; a.scale = (T)scale; a.vals = (T *)vals;
  return launch_tile<ScalarSpringTile<T>, T>(c, a, m);
}

template <typename T>
int heat(Ctx *c, const sg_mesh *m, const void *B, const void *W, const void *kappa, double dt,
         const void *T0, void *vals, void *b) {
  AsmArgs<T> a;
  fill_mesh(a, m);
  a.B = (const T *)B; a.W = (const T *)W; a.kappa = (const T *)kappa; a.dt = (T)dt;
  a.T0 = (const T *)T0; a.vals = (T *)vals; a.f = (T *)b;
  return launch_tile<HeatTile<T, SG_ASM_EXACT>, T>(c, a, m);
}

template <typename T>
int tet_precompute(Ctx *c, const sg_mesh *m, const void *x, double rho, void *B, void *W,
                   void *mass) {
  if (m->nE > 0) {
    k_tet_precompute<T><<<grid_for(c, m->nE, 128, 16), 128, 0, c->stream>>>(
        m->nE, m->endpoints, (const T *)x, (T *)B, (T *)W);
    SG_CHECK_LAUNCH();
  }
  AsmArgs<T> a;
  fill_mesh(a, m);
  a.W = (const T *)W; a.rho = (T)rho; a.f = (T *)mass;
  return launch_rows<TetMassElem<T>, 1, 1, T>(c, a);
}

template <typename T>
int blocks(Ctx *c, const sg_mesh *m, int bs, const void *eb, void *vals) {
  AsmArgs<T> a;
  fill_mesh(a, m);
  a.eb = (const T *)eb;
  a.vals = (T *)vals;
#define SG_BLK(BSV, CV)                                                            \
  if (bs == BSV && m->card == CV) {                                                \
    bool used = false;                                                             \
    SG_TRY((launch_plan<BSV, CV, T>(c, a, m, &used)));                             \
    if (used) return SG_OK;                                                        \
    return launch_rows<BlocksElem<T, BSV, CV>, 16, BSV, T>(c, a);                  \
  }
  SG_BLK(1, 2) SG_BLK(1, 3) SG_BLK(1, 4)
  SG_BLK(2, 2) SG_BLK(2, 3) SG_BLK(2, 4)
  SG_BLK(3, 2) SG_BLK(3, 3) SG_BLK(3, 4)
#undef SG_BLK
  return set_error(SG_ERR_UNSUPPORTED, "sg_assemble_blocks: bs %d, card %d (bs 1..3, card 2..4)",
                   bs, m->card);
}

template <typename T>
int tet_stiffness(Ctx *c, const sg_mesh *m, int model, const void *x, const int32_t *cons,
                  const void *B, const void *W, const void *mu, const void *lam, double h,
                  double rho, void *vals, void *eb_scratch) {
  AsmArgs<T> a;
  fill_mesh(a, m);
  a.x = (const T *)x; a.c = cons; a.B = (const T *)B; a.W = (const T *)W;
  a.mu = (const T *)mu; a.lam = (const T *)lam; a.h = (T)h; a.rho = (T)rho;
  a.vals = (T *)vals;
  if (!SG_ASM_EXACT)
    return model == SG_MODEL_NEOHOOKEAN ? launch_tile<NeoTile<T>, T>(c, a, m)
                                        : launch_tile<LinTetTile<T>, T>(c, a, m);
  if (model == SG_MODEL_NEOHOOKEAN) {
    a.eb = (const T *)eb_scratch;
    if (m->nE > 0) {
      k_neo_blocks<T><<<grid_for(c, m->nE, 128, 16), 128, 0, c->stream>>>(a);
      SG_CHECK_LAUNCH();
    }
    return launch_rows<EbGatherElem<T>, 16, 3, T>(c, a);
  }
  return launch_rows<LinTetElem<T>, 16, 3, T>(c, a);
}

template <typename T>
int tet_force(Ctx *c, const sg_mesh *m, int model, const void *x, const void *v,
              const int32_t *cons, const void *B, const void *W, const void *mu, const void *lam,
              double h, double rho, const double *grav, void *f) {
  AsmArgs<T> a;
  fill_mesh(a, m);
  a.x = (const T *)x; a.v = (const T *)v; a.c = cons; a.B = (const T *)B; a.W = (const T *)W;
  a.mu = (const T *)mu; a.lam = (const T *)lam; a.h = (T)h; a.rho = (T)rho;
  for (int q = 0; q < 3; ++q) a.grav[q] = (T)grav[q];
  a.f = (T *)f;
  if (!SG_ASM_EXACT)
    return model == SG_MODEL_NEOHOOKEAN ? launch_tile<TetForceTile<T, true>, T>(c, a, m)
                                        : launch_tile<TetForceTile<T, false>, T>(c, a, m);
  if (model == SG_MODEL_NEOHOOKEAN) return launch_rows<TetForceElem<T, true>, 4, 3, T>(c, a);
  return launch_rows<TetForceElem<T, false>, 4, 3, T>(c, a);
}

// Explicit instantiations for both precisions.
#define SG_INST(T)                                                                        \
  template int springs<T>(Ctx *, const sg_mesh *, int, const void *, const void *,       \
                          const void *, const uint8_t *, const void *, const void *, double, \
                          double, const double *, void *, void *);                       \
  template int scalar_springs<T>(Ctx *, const sg_mesh *, const void *, double, double,    \
                                 void *);                                                 \
  template int heat<T>(Ctx *, const sg_mesh *, const void *, const void *, const void *,   \
                       double, const void *, void *, void *);                             \
  template int tet_precompute<T>(Ctx *, const sg_mesh *, const void *, double, void *,    \
                                 void *, void *);                                         \
  template int blocks<T>(Ctx *, const sg_mesh *, int, const void *, void *);               \
  template int tet_stiffness<T>(Ctx *, const sg_mesh *, int, const void *, const int32_t *, \
                                const void *, const void *, const void *, const void *,   \
                                double, double, void *, void *);                          \
  template int tet_force<T>(Ctx *, const sg_mesh *, int, const void *, const void *,      \
                            const int32_t *, const void *, const void *, const void *,    \
                            const void *, double, double, const double *, void *);
SG_INST(float)
SG_INST(double)
#undef SG_INST

}  // namespace SG_ASM_NS
}  // namespace sg

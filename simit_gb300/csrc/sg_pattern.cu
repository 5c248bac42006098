// Pattern construction on the GPU: vertex incidence, blocked-CSR rows of
// ∃e∈E.(v-e ∧ e-u), and the element-to-slot map.
//
// Output is bit-identical to the reference's PathIndexBuilder
// (src/path_indices.cpp:148-531): row v is the sorted set of every endpoint
// of every element incident on v (empty when v has none), and slot (e,i,j)
// is the position `loc` (src/runtime.cpp:19-23) finds for
// (ep[e,i], ep[e,j]).
//
// Design: no std::set and no global sort.  Incidences are bucketed by vertex
// with integer atomics (counts only), and each vertex's bucket is then sorted
// by (e*card + i) inside one warp, so every result is deterministic.  Row
// columns: a warp per vertex puts the endpoints of its elements into a small
// shared-memory set and sorts what is left (a five-tet lattice row has 7 or 19
// columns among 32 or 128 endpoints), which is all the filling pass needs and
// more than the counting one does; slots from a binary search of the sorted
// row.
#include "sg_internal.cuh"

namespace sg {

__device__ __forceinline__ void dev_fail(int *err, int code) {
  atomicCAS(err, 0, code);
}

__global__ void inc_count(const int32_t *ep, int64_t m, int32_t n,
                          uint32_t *cnt, int *err) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < m;
       t += (int64_t)gridDim.x * blockDim.x) {
    int32_t v = ep[t];
    if (v < 0 || v >= n) {
      dev_fail(err, DEV_BAD_ENDPOINT);
      continue;
    }
    atomicAdd(&cnt[v], 1u);
  }
}

__global__ void inc_fill(const int32_t *ep, int64_t m, int32_t n,
                         uint32_t *cursor, uint32_t *ve_idx) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < m;
       t += (int64_t)gridDim.x * blockDim.x) {
    int32_t v = ep[t];
    if (v < 0 || v >= n) continue;
    uint32_t pos = atomicAdd(&cursor[v], 1u);
    ve_idx[pos] = (uint32_t)t;
  }
}

__global__ void max_u32_diff(const uint32_t *ptr, int32_t n, uint32_t *out) {
  uint32_t m = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    m = max(m, ptr[i + 1] - ptr[i]);
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_down_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// Warp-cooperative bitonic sort (ascending) of `len` (a power of two, >= 32)
// keys in shared memory.
__device__ void warp_bitonic_sort(uint32_t *s, int len) {
  const int lane = threadIdx.x & 31;
  for (int k = 2; k <= len; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = lane; i < len; i += 32) {
        int ixj = i ^ j;
        if (ixj > i) {
          uint32_t a = s[i], b = s[ixj];
          bool up = ((i & k) == 0);
          if ((a > b) == up) {
            s[i] = b;
            s[ixj] = a;
          }
        }
      }
      __syncwarp();
    }
  }
}

__device__ __forceinline__ int pow2_at_least(int x) {
  int p = 32;
  while (p < x) p <<= 1;
  return p;
}

// One warp per vertex: sort its incidence bucket ascending.
__global__ void inc_sort(const uint32_t *ve_ptr, uint32_t *ve_idx, int32_t n,
                         int cap, int *err) {
  extern __shared__ uint32_t smem[];
  const int wpb = blockDim.x >> 5;
  uint32_t *s = smem + (threadIdx.x >> 5) * cap;
  const int lane = threadIdx.x & 31;
  for (int64_t v = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); v < n;
       v += (int64_t)gridDim.x * wpb) {
    const uint32_t b = ve_ptr[v], e = ve_ptr[v + 1];
    const int len = (int)(e - b);
    if (len <= 1) continue;
    if (len <= 32) {  // register bitonic
      uint32_t key = lane < len ? ve_idx[b + lane] : 0xffffffffu;
      for (int k = 2; k <= 32; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
          uint32_t other = __shfl_xor_sync(0xffffffffu, key, j);
          bool up = ((lane & k) == 0);
          bool lower = ((lane & j) == 0);
          uint32_t mn = min(key, other), mx = max(key, other);
          key = (lower == up) ? mn : mx;
        }
      if (lane < len) ve_idx[b + lane] = key;
      continue;
    }
    if (len > cap) {
      if (lane == 0) dev_fail(err, DEV_ROW_TOO_LONG);
      continue;
    }
    const int p2 = pow2_at_least(len);
    for (int i = lane; i < p2; i += 32) s[i] = i < len ? ve_idx[b + i] : 0xffffffffu;
    __syncwarp();
    warp_bitonic_sort(s, p2);
    for (int i = lane; i < len; i += 32) ve_idx[b + i] = s[i];
    __syncwarp();
  }
}

// One warp per vertex: the distinct endpoints of its incident elements.  Pass 0
// writes their number to rowcnt[v], pass 1 the sorted columns at
// colidx[rowptr[v]...].  A row of more than SET_MAX distinct columns sets
// *over, and the caller runs rows_build.
//
// Bound by the gathers of the endpoints and shared-memory operations: at 64^3
// cells the passes take 114 and 141 us; sorting all 32..128 endpoints of
// every row in shared memory, twice, took 491 us a pass.
constexpr int MAX_SORT_CAP = 16384;  // keys per warp (64 KB) of rows_build and inc_sort
constexpr int SET_CAP = 256, SET_MAX = 192;  // table entries, columns kept
__global__ void __launch_bounds__(256) rows_set(const int32_t *ep, int32_t card,
                                                const uint32_t *ve_ptr, const uint32_t *ve_idx,
                                                int32_t n, int pass, uint32_t *rowcnt,
                                                const uint32_t *rowptr, uint32_t *colidx,
                                                uint32_t *over, int vec4) {
  __shared__ uint32_t tabs[8][SET_CAP], lists[8][SET_CAP];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *tab = tabs[warp], *list = lists[warp];
  for (int64_t v = (int64_t)blockIdx.x * 8 + warp; v < n; v += (int64_t)gridDim.x * 8) {
    const uint32_t b = ve_ptr[v], e = ve_ptr[v + 1];
    const int64_t len = (int64_t)(e - b) * card;
    int cap = 32;  // a table at most half full, if the row is short
    while (cap < SET_CAP && cap < 2 * len) cap <<= 1;
    for (int i = lane; i < cap; i += 32) tab[i] = 0xffffffffu;
    __syncwarp();
    // v itself is in every element of its row: it goes in once, ahead
    int cnt = len > 0 ? 1 : 0;
    if (lane == 0) list[0] = (uint32_t)v;
    bool full = len > MAX_SORT_CAP;  // (rows_build's limit, and its error)
    // a lane takes an incidence; its endpoints one after the other
    for (uint32_t k0 = b; k0 < e && !full; k0 += 32) {
      const uint32_t k = k0 + lane;
      const int64_t first = k < e ? (int64_t)(ve_idx[k] / (uint32_t)card) * card : -1;
      int4 four = make_int4(0, 0, 0, 0);
      if (vec4 && first >= 0) four = reinterpret_cast<const int4 *>(ep)[first / 4];
      for (int j = 0; j < card && !full; ++j) {
        uint32_t val = (uint32_t)v;
        if (first >= 0)
          val = (uint32_t)(!vec4 ? ep[first + j]
                                 : j == 0 ? four.x : j == 1 ? four.y : j == 2 ? four.z : four.w);
        bool fresh = false;
        if (val != (uint32_t)v) {
          uint32_t h = val * 0x9E3779B1u >> 16;
          for (;; ++h) {  // at most cnt + 32 <= SET_MAX + 32 entries are taken
            h &= (uint32_t)cap - 1u;
            const uint32_t old = atomicCAS(&tab[h], 0xffffffffu, val);
            fresh = old == 0xffffffffu;
            if (fresh || old == val) break;
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, fresh);
        if (fresh) list[cnt + __popc(m & ((1u << lane) - 1u))] = val;
        cnt += __popc(m);
        full = cnt > SET_MAX;
      }
    }
    __syncwarp();
    if (full) {
      if (lane == 0) atomicExch(over, 1u);
      if (pass == 0 && lane == 0) rowcnt[v] = 0;
      continue;
    }
    if (pass == 0) {
      if (lane == 0) rowcnt[v] = (uint32_t)cnt;
      continue;
    }
    uint32_t *out = colidx + rowptr[v];
    if (cnt <= 32) {  // register bitonic
      uint32_t key = lane < cnt ? list[lane] : 0xffffffffu;
      for (int k = 2; k <= 32; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
          const uint32_t other = __shfl_xor_sync(0xffffffffu, key, j);
          key = (((lane & j) == 0) == ((lane & k) == 0)) ? min(key, other) : max(key, other);
        }
      if (lane < cnt) out[lane] = key;
    } else {
      const int p2 = pow2_at_least(cnt);
      for (int i = cnt + lane; i < p2; i += 32) list[i] = 0xffffffffu;
      __syncwarp();
      warp_bitonic_sort(list, p2);
      for (int i = lane; i < cnt; i += 32) out[i] = list[i];
    }
    __syncwarp();
  }
}

// The same for rows of any length up to the sort capacity: gather the endpoints
// of every incident element, sort, unique.  Pass 0 writes the unique count to rowcnt[v]; pass 1 writes the
// columns at colidx[rowptr[v]...].
__global__ void rows_build(const int32_t *ep, int32_t card, const uint32_t *ve_ptr,
                           const uint32_t *ve_idx, int32_t n, int cap, int pass,
                           uint32_t *rowcnt, const uint32_t *rowptr,
                           uint32_t *colidx, int *err) {
  extern __shared__ uint32_t smem[];
  const int wpb = blockDim.x >> 5;
  uint32_t *s = smem + (threadIdx.x >> 5) * cap;
  const int lane = threadIdx.x & 31;
  for (int64_t v = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); v < n;
       v += (int64_t)gridDim.x * wpb) {
    const uint32_t b = ve_ptr[v], e = ve_ptr[v + 1];
    const int len = (int)(e - b) * card;
    if (len == 0) {
      if (pass == 0 && lane == 0) rowcnt[v] = 0;
      continue;
    }
    if (len > cap) {
      if (lane == 0) {
        dev_fail(err, DEV_ROW_TOO_LONG);
        if (pass == 0) rowcnt[v] = 0;
      }
      continue;
    }
    const int p2 = pow2_at_least(len);
    for (int i = lane; i < p2; i += 32) {
      uint32_t val = 0xffffffffu;
      if (i < len) {
        const uint32_t t = ve_idx[b + i / card];
        const uint32_t el = t / (uint32_t)card;
        val = (uint32_t)ep[(int64_t)el * card + (i % card)];
      }
      s[i] = val;
    }
    __syncwarp();
    warp_bitonic_sort(s, p2);
    // unique: keep s[i] when i == 0 or s[i] != s[i-1]
    uint32_t out = 0;
    const uint32_t base = (pass == 1) ? rowptr[v] : 0;
    for (int i0 = 0; i0 < len; i0 += 32) {
      const int i = i0 + lane;
      bool keep = (i < len) && (i == 0 || s[i] != s[i - 1]);
      unsigned mask = __ballot_sync(0xffffffffu, keep);
      if (pass == 1 && keep) colidx[base + out + __popc(mask & ((1u << lane) - 1))] = s[i];
      out += __popc(mask);
    }
    if (pass == 0 && lane == 0) rowcnt[v] = out;
    __syncwarp();
  }
}

// Thread per (e, i): the position of each ep[e, j] in row ep[e, i], four
// columns searched a step at a time so that their loads overlap.
__global__ void slots_build(const int32_t *ep, int64_t nE, int32_t card, int32_t n,
                           const uint32_t *rowptr, const uint32_t *colidx,
                           uint32_t *slots, int *err, int vec4) {
  const int64_t m = nE * card;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < m;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = t / card;
    const int32_t row = ep[t];
    if (row < 0 || row >= n) {
      dev_fail(err, DEV_BAD_ENDPOINT);
      for (int j = 0; j < card; ++j) slots[t * card + j] = 0xffffffffu;
      continue;
    }
    const uint32_t lo0 = rowptr[row], len = rowptr[row + 1] - lo0;
    uint32_t top = 1;  // the largest power of two <= len
    while (top <= len / 2) top *= 2;
    for (int j0 = 0; j0 < card; j0 += 4) {
      uint32_t col[4], lo[4];
      if (vec4) {
        const int4 f = reinterpret_cast<const int4 *>(ep)[e];
        col[0] = f.x; col[1] = f.y; col[2] = f.z; col[3] = f.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) col[j] = j0 + j < card ? (uint32_t)ep[e * card + j0 + j] : 0u;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) lo[j] = 0u;
      for (uint32_t st = top; st; st >>= 1) {  // lo: columns below col
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t q = lo[j] + st;
          if (q <= len && colidx[lo0 + q - 1] < col[j]) lo[j] = q;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j0 + j >= card) break;
        if (lo[j] >= len || colidx[lo0 + lo[j]] != col[j]) {
          dev_fail(err, DEV_SLOT_MISSING);
          lo[j] = 0xffffffffu;
        } else {
          lo[j] += lo0;
        }
      }
      if (vec4) {
        reinterpret_cast<uint4 *>(slots)[t] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j0 + j < card) slots[t * card + j0 + j] = lo[j];
      }
    }
  }
}

// Shared-memory capacity (keys per warp) for a maximum list length.
static int sort_cap(uint32_t maxlen) {
  int p = 32;
  while ((uint32_t)p < maxlen) p <<= 1;
  return p;
}

// The longest row to the context's staging word (valid after the next wait).
static int max_row_len_async(Ctx *c, uint32_t *d, const uint32_t *ptr, int32_t n) {
  SG_CHECK_CUDA(cudaMemsetAsync(d, 0, 4, c->stream));
  max_u32_diff<<<grid_for(c, n, 256, 4), 256, 0, c->stream>>>(ptr, n, d);
  SG_CHECK_LAUNCH();
  SG_CHECK_CUDA(cudaMemcpyAsync(c->h_stage, d, 4, cudaMemcpyDeviceToHost, c->stream));
  return SG_OK;
}

static int max_row_len(Ctx *c, Scratch &s, const uint32_t *ptr, int32_t n,
                       uint32_t *h_max) {
  SG_TRY(max_row_len_async(c, s.alloc<uint32_t>(1), ptr, n));
  SG_CHECK_CUDA(cudaStreamSynchronize(c->stream));
  *h_max = *(uint32_t *)c->h_stage;
  return SG_OK;
}

// Warps per block so that cap keys per warp fit the shared-memory budget.
static int warps_for_cap(int cap) {
  const int budget = 96 * 1024;
  int w = budget / (cap * 4);
  if (w > 8) w = 8;
  return w;
}

static int check_pattern_args(int32_t n, const int32_t *ep, int64_t nE, int32_t card) {
  SG_REQUIRE(n >= 0 && nE >= 0 && card >= 1 && card <= 64,
             "pattern: bad sizes n=%d nE=%lld card=%d", n, (long long)nE, card);
  SG_REQUIRE(nE == 0 || ep, "pattern: endpoints is null");
  SG_REQUIRE(nE * (int64_t)card < (int64_t)0xffffffffll,
             "pattern: nE*card must fit in uint32");
  return SG_OK;
}

}  // namespace sg

using namespace sg;

extern "C" {

int sg_incidence_build(sg_ctx *h, int32_t n, const int32_t *ep, int64_t nE,
                       int32_t card, uint32_t *ve_ptr, uint32_t *ve_idx) {
  Ctx *c = as_ctx(h);
  DeviceGuard dg_(c);
  SG_REQUIRE(c && ve_ptr && (nE == 0 || ve_idx), "sg_incidence_build: null argument");
  SG_TRY(check_pattern_args(n, ep, nE, card));
  const int64_t m = nE * card;
  Scratch s(c);
  SG_TRY(s.reserve(Scratch::bytes_for(n + 1, 4) * 2 + scan_scratch_bytes(n) + 1024));
  uint32_t *cnt = s.alloc<uint32_t>(n + 1);
  uint32_t *cursor = s.alloc<uint32_t>(n + 1);
  SG_CHECK_CUDA(cudaMemsetAsync(cnt, 0, (n + 1) * sizeof(uint32_t), c->stream));
  if (m > 0) {
    inc_count<<<grid_for(c, m, 256, 8), 256, 0, c->stream>>>(ep, m, n, cnt, c->d_err);
    SG_CHECK_LAUNCH();
  }
  SG_TRY(exclusive_scan_u32(c, s, cnt, ve_ptr, n));
  // the error word and the largest degree come back with one wait
  uint32_t *d_max = s.alloc<uint32_t>(1);
  SG_TRY(max_row_len_async(c, d_max, ve_ptr, n));
  SG_TRY(check_device_error(c, "sg_incidence_build"));
  if (m == 0) return SG_OK;
  const uint32_t maxdeg = *(uint32_t *)c->h_stage;
  SG_CHECK_CUDA(cudaMemcpyAsync(cursor, ve_ptr, n * sizeof(uint32_t),
                                cudaMemcpyDeviceToDevice, c->stream));
  inc_fill<<<grid_for(c, m, 256, 8), 256, 0, c->stream>>>(ep, m, n, cursor, ve_idx);
  SG_CHECK_LAUNCH();
  if (maxdeg > (uint32_t)MAX_SORT_CAP)
    return set_error(SG_ERR_UNSUPPORTED,
                     "sg_incidence_build: vertex degree %u exceeds %d", maxdeg, MAX_SORT_CAP);
  const int cap = sort_cap(maxdeg);
  const int w = warps_for_cap(cap);
  if ((size_t)w * cap * 4 > 48 * 1024)
    SG_CHECK_CUDA(cudaFuncSetAttribute(inc_sort, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       w * cap * 4));
  inc_sort<<<grid_for(c, (int64_t)n * 32, w * 32, 8), w * 32, (size_t)w * cap * 4, c->stream>>>(
      ve_ptr, ve_idx, n, cap, c->d_err);
  SG_CHECK_LAUNCH();
  return SG_OK;  // (cap holds the longest list: nothing left to check)
}

// rows_set; *over (cleared here) is set when a row has too many columns.
static int rows_set_launch(Ctx *c, const int32_t *ep, int32_t card, const uint32_t *ve_ptr,
                           const uint32_t *ve_idx, int32_t n, int pass, uint32_t *rowcnt,
                           const uint32_t *rowptr, uint32_t *colidx, uint32_t *over) {
  SG_CHECK_CUDA(cudaMemsetAsync(over, 0, 4, c->stream));
  rows_set<<<grid_for(c, (int64_t)n * 32, 256, 8), 256, 0, c->stream>>>(
      ep, card, ve_ptr, ve_idx, n, pass, rowcnt, rowptr, colidx, over,
      card == 4 && (uintptr_t)ep % 16 == 0);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

static int rows_launch(Ctx *c, Scratch &s, const int32_t *ep, int32_t card,
                       const uint32_t *ve_ptr, const uint32_t *ve_idx, int32_t n,
                       int pass, uint32_t *rowcnt, const uint32_t *rowptr,
                       uint32_t *colidx) {
  uint32_t maxdeg = 0;
  SG_TRY(max_row_len(c, s, ve_ptr, n, &maxdeg));
  const uint64_t maxlen = (uint64_t)maxdeg * card;
  if (maxlen > (uint64_t)MAX_SORT_CAP)
    return set_error(SG_ERR_UNSUPPORTED,
                     "sg_pattern: %llu candidate columns in one row exceed %d",
                     (unsigned long long)maxlen, MAX_SORT_CAP);
  const int cap = sort_cap((uint32_t)maxlen);
  const int w = warps_for_cap(cap);
  const size_t sh = (size_t)w * cap * 4;
  if (sh > 48 * 1024)
    SG_CHECK_CUDA(cudaFuncSetAttribute(rows_build,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh));
  rows_build<<<grid_for(c, (int64_t)n * 32, w * 32, 8), w * 32, sh, c->stream>>>(
      ep, card, ve_ptr, ve_idx, n, cap, pass, rowcnt, rowptr, colidx, c->d_err);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

int sg_pattern_count(sg_ctx *h, int32_t n, const int32_t *ep, int64_t nE,
                     int32_t card, const uint32_t *ve_ptr, const uint32_t *ve_idx,
                     uint32_t *rowptr, int64_t *h_nnzb) {
  Ctx *c = as_ctx(h);
  DeviceGuard dg_(c);
  SG_REQUIRE(c && ve_ptr && rowptr && h_nnzb, "sg_pattern_count: null argument");
  SG_TRY(check_pattern_args(n, ep, nE, card));
  Scratch s(c);
  SG_TRY(s.reserve(Scratch::bytes_for(n + 1, 4) + scan_scratch_bytes(n) + 1024));
  uint32_t *rowcnt = s.alloc<uint32_t>(n + 1);
  uint32_t *over = s.alloc<uint32_t>(1);
  uint32_t *hs = (uint32_t *)c->h_stage;
  SG_TRY(rows_set_launch(c, ep, card, ve_ptr, ve_idx, n, 0, rowcnt, nullptr, nullptr, over));
  for (int k = 0; k < 2; ++k) {
    Scratch t = s;  // (a second scan reuses the first one's scratch)
    SG_TRY(exclusive_scan_u32(c, t, rowcnt, rowptr, n));
    SG_CHECK_CUDA(cudaMemcpyAsync(hs, rowptr + n, 4, cudaMemcpyDeviceToHost, c->stream));
    SG_CHECK_CUDA(cudaMemcpyAsync(hs + 1, over, 4, cudaMemcpyDeviceToHost, c->stream));
    SG_TRY(check_device_error(c, "sg_pattern_count"));
    if (!hs[1] || k) break;
    SG_TRY(rows_launch(c, s, ep, card, ve_ptr, ve_idx, n, 0, rowcnt, nullptr, nullptr));
  }
  *h_nnzb = hs[0];
  return SG_OK;
}

int sg_pattern_fill(sg_ctx *h, int32_t n, const int32_t *ep, int64_t nE,
                    int32_t card, const uint32_t *ve_ptr, const uint32_t *ve_idx,
                    const uint32_t *rowptr, uint32_t *colidx) {
  Ctx *c = as_ctx(h);
  DeviceGuard dg_(c);
  SG_REQUIRE(c && ve_ptr && rowptr && (nE == 0 || colidx), "sg_pattern_fill: null argument");
  SG_TRY(check_pattern_args(n, ep, nE, card));
  Scratch s(c);
  SG_TRY(s.reserve(1024));
  uint32_t *over = s.alloc<uint32_t>(1);
  SG_TRY(rows_set_launch(c, ep, card, ve_ptr, ve_idx, n, 1, nullptr, rowptr, colidx, over));
  SG_CHECK_CUDA(cudaMemcpyAsync(c->h_stage, over, 4, cudaMemcpyDeviceToHost, c->stream));
  SG_TRY(check_device_error(c, "sg_pattern_fill"));
  if (!*(uint32_t *)c->h_stage) return SG_OK;
  SG_TRY(rows_launch(c, s, ep, card, ve_ptr, ve_idx, n, 1, nullptr, rowptr, colidx));
  return check_device_error(c, "sg_pattern_fill");
}

int sg_slots_build(sg_ctx *h, int32_t n, const int32_t *ep, int64_t nE,
                   int32_t card, const uint32_t *rowptr, const uint32_t *colidx,
                   uint32_t *slots) {
  Ctx *c = as_ctx(h);
  DeviceGuard dg_(c);
  SG_REQUIRE(c && rowptr && (nE == 0 || (colidx && slots)), "sg_slots_build: null argument");
  SG_TRY(check_pattern_args(n, ep, nE, card));
  const int64_t m = nE * card;
  if (m == 0) return SG_OK;
  slots_build<<<grid_for(c, m, 256, 8), 256, 0, c->stream>>>(
      ep, nE, card, n, rowptr, colidx, slots, c->d_err,
      card == 4 && (uintptr_t)ep % 16 == 0 && (uintptr_t)slots % 16 == 0);
  SG_CHECK_LAUNCH();
  return check_device_error(c, "sg_slots_build");
}

}  // extern "C"

// The window-grid path of one cloud (owm_grid.cuh): stage 1
// (optim3_func.cpp:541-561), stage 2 (:610-625) and stage 3 (:627-662) with
// their decisions on exact order keys, in seven launches:
//   k_grid_prepare   clears the tables, edge keys, s-ranges
//   k_grid_fold      every point into its sub-cell (count, (z, id)-min)
//   k_grid_rows      per sub-cell row and window column: reduce along x
//   k_grid_windows   per window: reduce along y, minNumPoints, stage 2's marks
//   k_grid_seeds     stage 2: count the ids marked twice, then write them in
//                    ascending order and mark the cells they lie in
//   k_grid_cells     stage 3: rectangle reduction of every unmarked cell
//   k_grid_output    stage-3 ids in cell order, then the LLPs
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "owm_devutil.cuh"
#include "owm_grid.cuh"

namespace owm {

namespace {

constexpr int kFoldBlock = 256;
constexpr int kFoldBlocks = 6;  // resident fold blocks per SM (40 registers a thread)

// ---- prepare ------------------------------------------------------------------
struct FormulaEdges {
  const GridAxis* a;
  __host__ __device__ __forceinline__ int64_t operator()(int f, int32_t j) const { return grid_edge(*a, f, j); }
};
struct StoredEdges {
  const GridAxis* a;
  __device__ __forceinline__ int64_t operator()(int f, int32_t j) const { return __ldg(a->edge[f] + j); }
};

__device__ int32_t class_of_key(const GridAxis& a, int64_t key) {
  int32_t cnt[4];
  grid_counts_exact(a, (uint64_t)__double_as_longlong(dkey_inv(key)), key, FormulaEdges{&a}, cnt);
  return grid_sum(a, cnt);
}

// Edge keys and s-ranges of item i of one axis (windows, then cells).
__device__ void prepare_axis(const GridAxis& a, int32_t i) {
  const bool win = i < a.n;
  const int32_t j = win ? i : i - a.n;
  const int f = win ? kFamL : kFamA;
  const int64_t l = grid_edge(a, f, j), r = grid_edge(a, f + 1, j);
  const_cast<int64_t*>(a.edge[f])[j] = l;
  const_cast<int64_t*>(a.edge[f + 1])[j] = r;
  if (!win && !a.merged) return;
  // no double lies between l and r when they touch: an empty range
  (win ? a.lo : a.clo)[j] = class_of_key(a, l + 1);
  (win ? a.hi : a.chi)[j] = l + 1 <= r - 1 ? class_of_key(a, r - 1) : -1;
}

// Bound by the stores of the clear (20 bytes a sub-cell, 2 bits a point);
// one launch instead of a memset and six small kernels.
__global__ void __launch_bounds__(256) k_grid_prepare(const __grid_constant__ GridJob J, uint4* __restrict__ clear,
                                                      int64_t nclear, uint32_t* __restrict__ status) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
  const int32_t nx = J.x.n + J.x.nc, ny = J.y.n + J.y.nc;
  for (int64_t i = t; i < nx + ny; i += nt) {
    if (i < nx) prepare_axis(J.x, (int32_t)i); else prepare_axis(J.y, (int32_t)i - nx);
  }
  if (t < 4) {
    const GridAxis& a = t < 2 ? J.x : J.y;
    J.occ[t] = !a.parmask || (t & 1) == 0;
  }
  if (t == 4) *status = 0;
  const uint4 z = make_uint4(0, 0, 0, 0);
  for (int64_t i = t; i < nclear; i += nt) clear[i] = z;
}

// ---- fold -----------------------------------------------------------------------
// Edge counts (L, R, A, B) of a coordinate outside the axis's [lo, hi].
__device__ __noinline__ int4 counts_outside(const GridAxis& a, uint64_t bits) {
  int32_t cnt[4];
  grid_counts_exact(a, bits, dkey(__longlong_as_double((long long)bits)), StoredEdges{&a}, cnt);
  return make_int4(cnt[0], cnt[1], cnt[2], cnt[3]);
}

__device__ __forceinline__ bool raw_finite(uint64_t b) { return ((uint32_t)(b >> 32) & 0x7FF00000u) != 0x7FF00000u; }

// Edge counts of a coordinate.  Coordinates in whole centimetres lie on an
// edge about once in 100; their edges are read side by side (loads that stay
// in L1) instead of one after the other in a call.
__device__ __forceinline__ int4 counts_of(const GridAxis& a, uint64_t bits) {
  int32_t c[4];
  if (grid_counts(a, bits, StoredEdges{&a}, c) == 2) return counts_outside(a, bits);
  return make_int4(c[0], c[1], c[2], c[3]);
}

__device__ __forceinline__ int32_t class_of(const GridAxis& a, const int4& c) {
  return c.x + c.y + (a.merged ? c.z + c.w : 0);
}

__device__ __forceinline__ ulonglong2 load_zid(const ulonglong2* p) {
  ulonglong2 r;
  asm volatile("{\n\t.reg .b128 v;\n\tld.relaxed.gpu.global.b128 v, [%2];\n\tmov.b128 {%0, %1}, v;\n\t}"
               : "=l"(r.x), "=l"(r.y)
               : "l"(p));
  return r;
}

__device__ __forceinline__ bool zid_above(unsigned long long w, uint32_t nid, const ulonglong2& e) {
  return w > e.x || (w == e.x && nid > e.y);
}

// Raises *p to (w, nid) if that is above it; cur is what *p held (a value
// read earlier only makes the first swap fail).  The stored pair only rises
// and a failed swap means that another thread raised it, so the loop ends.
__device__ __forceinline__ void raise_zid(ulonglong2* p, ulonglong2 cur, unsigned long long w, uint32_t nid) {
  while (zid_above(w, nid, cur)) {
    ulonglong2 old;
    asm volatile(
        "{\n\t.reg .b128 d, b, c;\n\t"
        "mov.b128 b, {%2, %3};\n\t"
        "mov.b128 c, {%4, %5};\n\t"
        "atom.relaxed.gpu.global.cas.b128 d, [%6], b, c;\n\t"
        "mov.b128 {%0, %1}, d;\n\t}"
        : "=l"(old.x), "=l"(old.y)
        : "l"(cur.x), "l"(cur.y), "l"(w), "l"((unsigned long long)nid), "l"(p)
        : "memory");
    if (old.x == cur.x && old.y == cur.y) break;
    cur = old;
  }
}

// Point i as raw bits, read once: 32-byte records or plain 24-byte points.
template <int kStride>
__device__ __forceinline__ void load_raw(const double* __restrict__ rec, int64_t i, uint64_t& x, uint64_t& y, uint64_t& z) {
  if (kStride == 4) {
    asm("ld.global.nc.L1::no_allocate.L2::evict_first.v4.b64 {%0, %1, %2, _}, [%3];"
        : "=l"(x), "=l"(y), "=l"(z)
        : "l"(rec + 4 * i));
  } else {
    const uint64_t* p = reinterpret_cast<const uint64_t*>(rec) + 3 * i;
    x = __ldg(p);
    y = __ldg(p + 1);
    z = __ldg(p + 2);
  }
}

// Inverted, sign-flipped order key of the double with these bits (-0 as +0).
__device__ __forceinline__ unsigned long long inverted_key(uint64_t b) {
  if (b == 0x8000000000000000ull) b = 0;
  return (int64_t)b < 0 ? b : ~b & 0x7FFFFFFFFFFFFFFFull;
}

struct PointCell {
  unsigned long long w;  // inverted key of z
  uint32_t cell, flags;
};
constexpr uint32_t kPointOtherX = 1, kPointOtherY = 2, kPointNonFinite = 4;

// A point's sub-cell and z, in full: any coordinate, any axes.
__device__ __forceinline__ PointCell point_cell(const GridJob& J, uint64_t x, uint64_t y, uint64_t z) {
  PointCell p;
  const int32_t sx = class_of(J.x, counts_of(J.x, x)), sy = class_of(J.y, counts_of(J.y, y));
  p.w = inverted_key(z);
  p.cell = grid_cell(J, sx, sy);
  p.flags = (((sx ^ J.x.par) & J.x.parmask) ? kPointOtherX : 0u) | (((sy ^ J.y.par) & J.y.parmask) ? kPointOtherY : 0u) |
            (raw_finite(x) & raw_finite(y) & raw_finite(z) ? 0u : kPointNonFinite);
  return p;
}
__device__ __noinline__ PointCell point_cell_call(const GridJob& J, uint64_t x, uint64_t y, uint64_t z) {
  return point_cell(J, x, y, z);
}

// The point into the cells that are not merged (rarely more than one).
__device__ __noinline__ void raise_own_cells(const GridJob& J, uint64_t x, uint64_t y, unsigned long long w, uint32_t nid) {
  const int4 cx = counts_of(J.x, x), cy = counts_of(J.y, y);
  for (int32_t cj = cy.w; cj < cy.z; ++cj)
    for (int32_t ci = cx.w; ci < cx.z; ++ci) {
      ulonglong2* p = J.cell_zid + (int64_t)cj * J.x.nc + ci;
      raise_zid(p, load_zid(p), w, nid);
    }
}

// Every point into its sub-cell.  kFast: both axes have the fast form, and
// whatever it does not settle (an edge, a point outside the box, z zero or not
// finite) takes the full one in a call.
//
// Bound by the L2 requests of points in no order (a read and an add each): 100 M
// points into 0.9 M sub-cells take 1.04 ms (32 bytes a point: 3.1 TB/s), a bare
// kernel that does just those two requests 0.87.  The order of the work and the
// instructions were what cost before: a warp takes a stretch of neighbouring
// points, so that scan lines side by side are not folded at the same time (40 M
// points in scan order at 3 a square metre: 1.28 -> 0.53 ms); 144 instructions
// per 32 points instead of 284 (0.53 -> 0.40); one point a thread at 48 warps
// an SM (two at 40: 1.05 ms for the 100 M, four at 32: 1.05, and 0.40 -> 0.46
// for the scan).  A single add whose result carries a filter for the minimum
// measured 1.40 ms at 100 M.
template <int kStride, bool kFast>
__global__ void __launch_bounds__(kFoldBlock, kFoldBlocks)
    k_grid_fold(const __grid_constant__ GridJob J, const double* __restrict__ rec, int64_t first, int64_t count,
                uint32_t* __restrict__ status) {
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = ((int64_t)gridDim.x * kFoldBlock) >> 5;
  uint32_t flags = 0;
  int64_t t0, t1;
  chunk_tiles((count + 31) / 32, nwarps, ((int64_t)blockIdx.x * kFoldBlock + threadIdx.x) >> 5, &t0, &t1);
  for (int64_t b = t0 * 32; b < t1 * 32; b += 32) {
    // lanes past the end take the last point again, and are not counted
    const int32_t left = (int32_t)min((int64_t)32, count - b);
    const int64_t i = first + b + min(lane, left - 1);
    uint64_t x, y, z;
    load_raw<kStride>(rec, i, x, y, z);
    uint32_t cell, nid = ~(uint32_t)(i + 1);
    unsigned long long w;
    if (kFast) {
      bool rare = ((uint32_t)(z >> 32) << 1) - 1u >= 0xFFDFFFFFu;  // zero or not finite
      const int32_t sx = grid_class_fast(J.x, x, &rare), sy = grid_class_fast(J.y, y, &rare);
      rare |= ((sx ^ J.x.par) | (sy ^ J.y.par)) & 1;
      cell = (uint32_t)(sy >> 1) * (uint32_t)J.x.width[0] + (uint32_t)(sx >> 1);
      w = z ^ (~(uint64_t)((int64_t)z >> 63) & 0x7FFFFFFFFFFFFFFFull);
      if (rare) {
        const PointCell p = point_cell_call(J, x, y, z);
        cell = p.cell;
        w = p.w;
        flags |= p.flags;
      }
    } else {
      const PointCell p = point_cell(J, x, y, z);
      cell = p.cell;
      w = p.w;
      flags |= p.flags;
      if (J.cell_zid) raise_own_cells(J, x, y, w, nid);
    }
    const ulonglong2 cur = load_zid(J.zid + cell);
    // runs of neighbouring lanes in one sub-cell (a cloud in scan order)
    const uint32_t before = __shfl_up_sync(0xffffffffu, cell, 1);
    const uint32_t heads = __ballot_sync(0xffffffffu, before != cell) | 1u;
    if (heads == 0xFFFFFFFFu) {  // none (a lane past the end would repeat its neighbour)
      atomicAdd(J.count + cell, 1u);
      if (w >= cur.x) raise_zid(J.zid + cell, cur, w, nid);
      continue;
    }
    const uint32_t after = heads & (0xFFFFFFFEu << lane);
    const int end = after ? __ffs(after) - 1 : 32;
    const bool head = (heads >> lane) & 1u;
    const int run = min(end, left) - lane;
    if (head && run > 0) atomicAdd(J.count + cell, (uint32_t)run);
    if (!__any_sync(0xffffffffu, w >= cur.x)) continue;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {  // the run's minimum, to its head
      const unsigned long long ow = __shfl_down_sync(0xffffffffu, w, o);
      const uint32_t on = __shfl_down_sync(0xffffffffu, nid, o);
      if (lane + o < end && (ow > w || (ow == w && on > nid))) {
        w = ow;
        nid = on;
      }
    }
    if (head) raise_zid(J.zid + cell, cur, w, nid);
  }
  // one store a warp: a store per point to the one word cost 0.4 ms on 40 M
  // points in whole centimetres
  flags = __reduce_or_sync(0xffffffffu, flags);
  if (lane == 0 && flags) {
    if (flags & kPointNonFinite) atomicOr(status, kStatusNonFinite);
    if (flags & kPointOtherX) J.occ[1] = 1;
    if (flags & kPointOtherY) J.occ[3] = 1;
  }
}

// ---- rectangle reductions ---------------------------------------------------------
struct Best {
  unsigned long long w = 0;
  uint32_t nid = 0, count = 0;
  __device__ __forceinline__ void take(unsigned long long ow, uint32_t onid) {
    if (ow > w || (ow == w && onid > nid)) {
      w = ow;
      nid = onid;
    }
  }
};

// First and last s >> 1 of the classes lo..hi of the main (q = 0) or the other
// parity; false when there are none or they hold no point.
__device__ __forceinline__ bool parity_range(const GridAxis& a, const uint32_t* occ, int q, int32_t lo, int32_t hi,
                                             int32_t* i0, int32_t* i1) {
  if (!occ[q]) return false;
  const int32_t par = a.par ^ q, s0 = lo + ((lo ^ par) & 1), s1 = hi - ((hi ^ par) & 1);
  if (s0 > s1) return false;
  *i0 = s0 >> 1;
  *i1 = s1 >> 1;
  return true;
}

__global__ void __launch_bounds__(256) k_grid_rows(const __grid_constant__ GridJob J) {
  const int64_t total = (int64_t)J.y.nclass * J.x.n;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (int64_t)gridDim.x * blockDim.x) {
    const int32_t r = (int32_t)(k / J.x.n), ii = (int32_t)(k % J.x.n);
    const int qy = r >= J.y.width[0];
    if (!J.occ[2 + qy]) continue;
    const int32_t iy = r - (qy ? J.y.width[0] : 0), lo = J.x.lo[ii], hi = J.x.hi[ii];
    Best m;
    for (int q = 0; q < 2; ++q) {
      int32_t i0, i1;
      if (!parity_range(J.x, J.occ, q, lo, hi, &i0, &i1)) continue;
      const int64_t at = J.base[2 * qy + q] + (int64_t)iy * J.x.width[q];
      for (int64_t c = at + i0; c <= at + i1; ++c) {
        const ulonglong2 e = J.zid[c];
        m.count += J.count[c];
        m.take(e.x, (uint32_t)e.y);
      }
    }
    GridRow o;
    o.w = m.w;
    o.nid = m.nid;
    o.count = m.count;
    J.rows[k] = o;
  }
}

__global__ void __launch_bounds__(256) k_grid_windows(const __grid_constant__ GridJob J) {
  // the search starts from the reference's sentinel point 0 {0, 0, DBL_MAX}
  const unsigned long long sentinel = ~((unsigned long long)kZSentinel ^ 0x8000000000000000ull);
  const int64_t total = (int64_t)J.x.n * J.y.n;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (int64_t)gridDim.x * blockDim.x) {
    const int32_t jj = (int32_t)(k / J.x.n), ii = (int32_t)(k % J.x.n);
    Best m;
    m.w = sentinel;
    m.nid = ~0u;
    for (int q = 0; q < 2; ++q) {
      int32_t i0, i1;
      if (!parity_range(J.y, J.occ + 2, q, J.y.lo[jj], J.y.hi[jj], &i0, &i1)) continue;
      const int64_t at = q ? J.y.width[0] : 0;
      for (int32_t r = i0; r <= i1; ++r) {
        const GridRow e = J.rows[(at + r) * J.x.n + ii];
        m.count += e.count;
        m.take(e.w, e.nid);
      }
    }
    const uint32_t id = m.count >= J.thr ? ~m.nid : kNone;
    if (J.win)
      J.win[(int64_t)ii * J.y.n + jj] = id;
    else
      s2_mark_id(J.once, J.twice, (uint32_t)J.n, id);
  }
}

// ---- stage 2 ------------------------------------------------------------------
constexpr int kSeedBlock = 256;
constexpr int kSeedWords = 4;
constexpr int64_t kSeedChunk = (int64_t)kSeedBlock * kSeedWords;  // bitmap words a block takes

__device__ __forceinline__ uint32_t block_exclusive_256(uint32_t v, uint32_t* total) {
  __shared__ uint32_t ws[kSeedBlock / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  __syncthreads();  // the last call's readers of ws are done
  if (lane == 31) ws[w] = inc;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int q = 0; q < kSeedBlock / 32; ++q) {
    const uint32_t x = ws[q];
    before += q < w ? x : 0u;
    all += x;
  }
  *total = all;
  return before + inc - v;
}

__global__ void __launch_bounds__(kSeedBlock) k_grid_seed_count(const uint32_t* __restrict__ bm, uint32_t* __restrict__ part) {
  const uint4 q = __ldg(reinterpret_cast<const uint4*>(bm) + (int64_t)blockIdx.x * kSeedBlock + threadIdx.x);
  uint32_t total;
  block_exclusive_256((uint32_t)(__popc(q.x) + __popc(q.y) + __popc(q.z) + __popc(q.w)), &total);
  if (threadIdx.x == 0) part[blockIdx.x] = total;
}

// Marks the stage-3 cells that hold LLP `id` strictly inside (the LLP grid,
// owm_optim3.cpp:192-197); id 0 is the sentinel point {0, 0, DBL_MAX}.
__device__ __forceinline__ void mark_cells(const GridJob& J, const double* __restrict__ xy, int stride, uint32_t id) {
  uint64_t x = 0, y = 0;
  if (id > 0) {
    const uint64_t* p = reinterpret_cast<const uint64_t*>(xy) + stride * (int64_t)(id - 1);
    x = __ldg(p);
    y = __ldg(p + 1);
  }
  const int4 cx = counts_of(J.x, x), cy = counts_of(J.y, y);
  for (int32_t cj = cy.w; cj < cy.z; ++cj)
    for (int32_t ci = cx.w; ci < cx.z; ++ci) J.mark[(int64_t)cj * J.x.nc + ci] = 1;
}

// The ids marked twice, ascending: block b writes those of its chunk after
// all chunks before it (whose counts it adds up) and marks their cells.
__global__ void __launch_bounds__(kSeedBlock) k_grid_seeds(const __grid_constant__ GridJob J, const uint32_t* __restrict__ part,
                                                           const double* __restrict__ xy, int stride,
                                                           uint32_t* __restrict__ llp, uint32_t* __restrict__ nllp) {
  uint32_t before = 0, total;
  for (uint32_t q = threadIdx.x; q < blockIdx.x; q += kSeedBlock) before += __ldg(part + q);
  block_exclusive_256(before, &before);
  const int64_t w0 = (int64_t)blockIdx.x * kSeedChunk + (int64_t)threadIdx.x * kSeedWords;
  const uint4 q = __ldg(reinterpret_cast<const uint4*>(J.twice + w0));
  const uint32_t word[4] = {q.x, q.y, q.z, q.w};
  uint32_t at = before + block_exclusive_256((uint32_t)(__popc(q.x) + __popc(q.y) + __popc(q.z) + __popc(q.w)), &total);
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *nllp = before + total;
#pragma unroll
  for (int k = 0; k < kSeedWords; ++k) {
    uint32_t b = word[k];
    while (b) {
      const uint32_t id = (uint32_t)((w0 + k) * 32) + (uint32_t)(__ffs(b) - 1);
      b &= b - 1;
      llp[at++] = id;
      if (J.x.nc) mark_cells(J, xy, stride, id);
    }
  }
}

// The cells of LLPs that another kernel listed.
__global__ void __launch_bounds__(256) k_grid_mark(const __grid_constant__ GridJob J, const double* __restrict__ xy, int stride,
                                                   const uint32_t* __restrict__ llp, const uint32_t* __restrict__ nllp) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < *nllp; k += gridDim.x * blockDim.x)
    mark_cells(J, xy, stride, llp[k]);
}

// ---- stage 3 ----------------------------------------------------------------------
// Result of a cell from its minimum (w 0: no point).  The reference's search
// starts from the sentinel {0, 0, DBL_MAX}: a cell whose points all lie at
// DBL_MAX keeps id 0.
__device__ __forceinline__ uint32_t cell_result(unsigned long long w, uint32_t nid) {
  const unsigned long long sentinel = ~((unsigned long long)kZSentinel ^ 0x8000000000000000ull);
  return w == 0 ? kNone : w <= sentinel ? 0u : ~nid;
}

// One warp per cell: the (z, id)-min of its rectangle of sub-cells.
__global__ void __launch_bounds__(256) k_grid_cells(const __grid_constant__ GridJob J, int64_t ncell) {
  const int lane = threadIdx.x & 31;
  const int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= ncell) return;
  const int32_t ci = (int32_t)(c % J.x.nc), cj = (int32_t)(c / J.x.nc);
  Best m;
  if (!J.mark[c]) {
    for (int qy = 0; qy < 2; ++qy) {
      int32_t y0, y1;
      if (!parity_range(J.y, J.occ + 2, qy, J.y.clo[cj], J.y.chi[cj], &y0, &y1)) continue;
      for (int qx = 0; qx < 2; ++qx) {
        int32_t x0, x1;
        if (!parity_range(J.x, J.occ, qx, J.x.clo[ci], J.x.chi[ci], &x0, &x1)) continue;
        const int32_t nx = x1 - x0 + 1, tot = nx * (y1 - y0 + 1);
        const int64_t at = J.base[2 * qy + qx] + x0;
        for (int32_t k = lane; k < tot; k += 32) {
          const ulonglong2 e = J.zid[at + (int64_t)(y0 + k / nx) * J.x.width[qx] + k % nx];
          m.take(e.x, (uint32_t)e.y);
        }
      }
    }
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1)
    m.take(__shfl_xor_sync(0xffffffffu, m.w, o), __shfl_xor_sync(0xffffffffu, m.nid, o));
  if (lane == 0) J.cellmin[c] = cell_result(m.w, m.nid);
}

__global__ void __launch_bounds__(256) k_grid_cells_own(const __grid_constant__ GridJob J, int64_t ncell) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  const ulonglong2 e = J.cell_zid[c];
  J.cellmin[c] = J.mark[c] ? kNone : cell_result(e.x, (uint32_t)e.y);
}

// seeds = the valid entries of cellmin in order, then the LLPs.  Every block
// counts all cells (at most kOutputCells) for the total and its own start.
constexpr int64_t kOutputCells = 32768;
__global__ void __launch_bounds__(kSeedBlock) k_grid_output(const uint32_t* __restrict__ cellmin, int64_t ncell,
                                                            const uint32_t* __restrict__ llp, const uint32_t* __restrict__ nllp,
                                                            int64_t* __restrict__ seeds, uint32_t* __restrict__ ns3) {
  const int64_t per = (ncell + gridDim.x - 1) / gridDim.x;
  const int64_t b0 = per * blockIdx.x, b1 = min(b0 + per, ncell);
  uint32_t before = 0, all = 0;
  for (int64_t i = threadIdx.x; i < ncell; i += kSeedBlock) {
    const uint32_t v = __ldg(cellmin + i) != kNone ? 1u : 0u;
    all += v;
    if (i < b0) before += v;
  }
  block_exclusive_256(before, &before);
  block_exclusive_256(all, &all);
  if (blockIdx.x == 0 && threadIdx.x == 0) *ns3 = all;
  uint32_t at = before;
  for (int64_t t = b0; t < b1; t += kSeedBlock) {
    const uint32_t v = t + threadIdx.x < b1 ? __ldg(cellmin + t + threadIdx.x) : kNone;
    uint32_t got;
    const uint32_t p = block_exclusive_256(v != kNone ? 1u : 0u, &got);
    if (v != kNone) seeds[at + p] = v;
    at += got;
  }
  const uint32_t n = *nllp;
  for (uint32_t k = blockIdx.x * kSeedBlock + threadIdx.x; k < n; k += gridDim.x * kSeedBlock) seeds[all + k] = llp[k];
}

__global__ void k_grid_flags(const uint32_t* __restrict__ v, int64_t n, uint32_t* __restrict__ flags) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    flags[i] = v[i] != kNone ? 1u : 0u;
}
__global__ void k_grid_output_scanned(const uint32_t* __restrict__ cellmin, const uint32_t* __restrict__ pos, int64_t ncell,
                                      const uint32_t* __restrict__ llp, const uint32_t* __restrict__ nllp,
                                      const uint32_t* __restrict__ ns3, int64_t* __restrict__ seeds) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = t; i < ncell; i += nt)
    if (cellmin[i] != kNone) seeds[pos[i]] = cellmin[i];
  const int64_t n = *nllp, base = *ns3;
  for (int64_t i = t; i < n; i += nt) seeds[base + i] = llp[i];
}

unsigned blocks_for(int64_t n, int64_t most, int block = 256) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + block - 1) / block, most));
}

size_t up256(size_t b) { return (b + 255) & ~(size_t)255; }

int64_t bits_of(double d) {
  int64_t b;
  std::memcpy(&b, &d, 8);
  return b;
}

int64_t quanta_of(double v, int sh) {  // grid_position's general form
  const uint64_t bits = (uint64_t)bits_of(v);
  const int e = (int)((bits >> 52) & 0x7FF);
  const uint64_t m = (bits & 0xFFFFFFFFFFFFFull) | (e ? 0x10000000000000ull : 0ull);
  const int s = sh - (e ? e : 1);
  const int64_t f = s > 63 ? 0 : (int64_t)(m >> s);
  return v < 0 ? -f : f;
}

// Constants of one pair of families (first edges l0 <= r0, n of each at every
// step) over positions of qv each from origin; false when a place has too few
// fraction bits.
bool place_setup(double origin, double qv, double l0, double r0, double step, uint32_t* m, uint32_t* cl, uint32_t* cr,
                 int32_t* fb, int32_t* bias) {
  const double k = std::max(0.0, std::ceil((r0 - origin) / step)) + 1.0;
  const double most = (origin + std::ldexp(qv, 32) - l0) / step + k + 3.0;
  if (!(most > 0.0) || !(std::ldexp(most, kGridMinFrac) <= 4294967296.0)) return false;
  int f = 30;
  while (std::ldexp(most, f) > 4294967296.0) --f;
  *m = (uint32_t)(std::ldexp(qv / step, 32 + f) + 0.5);
  *cl = (uint32_t)(std::ldexp(k + 1.0 + (origin - l0) / step, f) + 0.5) + kGridGuard;
  *cr = (uint32_t)(std::ldexp(k + 1.0 + (origin - r0) / step, f) + 0.5) + kGridGuard;
  *fb = f;
  *bias = (int32_t)k;
  return true;
}

}  // namespace

void grid_axis_setup(double lo, double hi, double step, int32_t whalf, int32_t n, int32_t bsize, int32_t nc, bool merged,
                     GridAxis* a) {
  std::memset(a, 0, sizeof(*a));
  a->n = n;
  a->nc = nc;
  a->bsize = bsize;
  a->step = step;
  a->wbase = (lo - (double)whalf) + step;
  a->wr = (double)(float)whalf;
  const int32_t chalf = bsize / 2;
  a->cbase = lo + (double)chalf;
  a->cr = (double)(float)chalf;
  a->merged = merged ? 1 : 0;
  a->nclass = 2 * n + (merged ? 2 * nc : 0) + 1;
  // no cells: a place that passes no edge and is near none
  a->fbc = 30;
  a->c[kFamA] = a->c[kFamB] = 4 * kGridGuard;
  a->linear = 1;

  const double span = hi - lo;
  double origin = 0.0, qv = 0.0;
  bool quick = std::isfinite(span) && span > 0.0;
  bool linear = false;
  if (quick && lo > 0.0) {
    const int64_t bl = bits_of(lo), bh = bits_of(hi), e = bl >> 52;
    int len = 0;
    while (((uint64_t)(bh - bl) >> len) != 0) ++len;
    const int sh = std::max(0, len - 31);
    const int64_t f0 = bl - ((int64_t)1 << (30 + sh)), top = f0 + ((int64_t)1 << (32 + sh)) - 1;
    if (e >= 1 && e == (bh >> 52) && f0 > 0 && (f0 >> 52) == e && (top >> 52) == e) {
      linear = true;
      a->f0 = f0;
      a->sh = sh;
      std::memcpy(&origin, &f0, 8);
      qv = std::ldexp(1.0, (int)e - 1075 + sh);
    }
  }
  if (quick && !linear) {
    const double big = std::max(std::fabs(lo), std::fabs(hi));
    int q = std::max(std::ilogb(span) - 30, -1074);
    while (q < std::ilogb(big + std::ldexp(1.0, q + 32)) - 52) ++q;
    a->linear = 0;
    a->sh = q + 1075;
    a->f0 = quanta_of(lo, a->sh) - ((int64_t)1 << 30);
    origin = std::ldexp((double)a->f0, q);
    qv = std::ldexp(1.0, q);
    quick = std::isfinite(origin) && std::isfinite(std::ldexp(qv, 33));
  }
  if (quick) {
    const double c0 = a->wbase, l0 = c0 - a->wr, r0 = c0 + a->wr;
    quick = place_setup(origin, qv, l0, r0, step, &a->mw, &a->c[kFamL], &a->c[kFamR], &a->fbw, &a->kw);
    if (quick && nc > 0)
      quick = place_setup(origin, qv, a->cbase - a->cr, a->cbase + a->cr, (double)bsize, &a->mc, &a->c[kFamA], &a->c[kFamB],
                          &a->fbc, &a->kc);
  }
  a->quick = quick ? 1 : 0;
  // the fast form, from lo; an empty range (span 0 above the greatest position) without one
  a->lo0 = linear ? bits_of(lo) : 0;
  a->span = 0;
  if (quick) {
    const double step2 = (double)bsize, at = linear ? lo : origin + std::ldexp(qv, 30);
    auto place = [](double from, double l0, double st, int32_t fb, int32_t k) {
      return (uint32_t)(std::ldexp(k + 1.0 + (from - l0) / st, fb) + 0.5) + kGridGuard;
    };
    const double l0 = a->wbase - a->wr, r0 = a->wbase + a->wr;
    a->qw = place(at, l0, step, a->fbw, a->kw);
    a->qr = place(at, r0, step, a->fbw, a->kw);
    a->kl = a->kr = a->kw;
    a->qc = a->c[kFamA];
    a->qb = a->c[kFamB];
    bool pair = true;
    // one place for both families when their places differ by whole steps
    // (and at most 4 units, which the guard has to spare)
    auto merge = [&](uint32_t q0, uint32_t q1, int32_t fb, int32_t* k1) {
      const int64_t d = (int64_t)q0 - q1, steps = (d + ((int64_t)1 << (fb - 1))) >> fb;
      if (std::llabs(d - (steps << fb)) > 4) return false;
      *k1 += (int32_t)steps;
      return true;
    };
    int32_t kr = a->kr, kb = a->kc;
    pair = merge(a->qw, a->qr, a->fbw, &kr);
    if (nc > 0) {
      a->qc = place(at, a->cbase - a->cr, step2, a->fbc, a->kc);
      a->qb = place(at, a->cbase + a->cr, step2, a->fbc, a->kc);
      pair = merge(a->qc, a->qb, a->fbc, &kb) && pair;
    }
    a->ka = a->kb = a->kc;
    a->paired = pair ? 1 : 0;
    if (pair) {
      a->kr = kr;
      a->kb = kb;
    }
    a->span = linear ? (uint64_t)(bits_of(hi) - bits_of(lo)) : (uint64_t)(quanta_of(hi, a->sh) - quanta_of(lo, a->sh));
  } else {
    a->linear = 1;  // no finite double lies at its range
    a->lo0 = (int64_t)0xFFFFFFFFFFFFFFFFull;
    a->sh = 0;
  }
  // Whether every right edge nominally coincides with a left one (and the
  // cells' edges with one another): then the classes off the edges are all of
  // one parity, which is read off the middle of the axis.  Only a hint: a
  // point of the other parity says so in J.occ.
  const double steps = 2.0 * whalf / step;
  if (std::fabs(steps - std::round(steps)) < 1e-6 && (!merged || nc == 0 || bsize % 2 == 0)) {
    int32_t cnt[4];
    const double mid = lo + 0.4637 * span;
    grid_counts_exact(*a, (uint64_t)bits_of(mid), dkey(mid), FormulaEdges{a}, cnt);
    a->par = grid_sum(*a, cnt) & 1;
    a->parmask = 1;
  }
  const int32_t even = (a->nclass + 1) / 2;
  a->width[0] = a->par ? a->nclass - even : even;
  a->width[1] = a->nclass - a->width[0];
  if (a->paired && a->linear && a->parmask && (merged || nc == 0)) {
    a->lcap = n + a->kl;
    a->ksum = a->kl + a->kr + a->ka + a->kb;
    int32_t at_lo[4], at_hi[4];  // no clamps but the left windows' upper one
    const int how0 = grid_counts_raw(*a, (uint64_t)bits_of(lo), at_lo), how1 = grid_counts_raw(*a, (uint64_t)bits_of(hi), at_hi);
    a->fast = how0 != 2 && how1 != 2 && at_hi[1] <= n && at_hi[2] <= nc && at_hi[3] <= nc;
    for (int f = 0; f < 4; ++f) a->fast = a->fast && at_lo[f] >= -how0;
  }
}

int grid_plan(const owm_params& p, int64_t n, void* scratch, GridPlan* g) {
  *g = GridPlan{};
  GridJob& J = g->job;
  std::memset(&J, 0, sizeof(J));
  const int32_t nc = (int32_t)p.ncols, nr = (int32_t)p.nrows;
  if (nc <= 0 || nr <= 0) return OWM_EINVAL;
  const int64_t tx = 2 * (int64_t)nc + 1, ty = 2 * (int64_t)nr + 1;
  if (tx * ty >= 0xFFFFFFFFll) return OWM_ERANGE;
  const bool cells = p.bsize > 0 && p.ngrid > 0;
  const int32_t ncg = cells ? (int32_t)p.ncols_grid : 0, nrg = cells ? (int32_t)p.nrows_grid : 0;
  const bool merged = cells && (tx + 2 * ncg) * (ty + 2 * nrg) <= std::min<int64_t>(std::max<int64_t>(4 * tx * ty, 1 << 20), 1 << 28);
  const int32_t whalf = (uint16_t)p.wsize / 2, bsize = (uint16_t)p.bsize;
  grid_axis_setup(p.bbox.min_x, p.bbox.max_x, p.displace, whalf, nc, bsize, ncg, merged, &J.x);
  grid_axis_setup(p.bbox.min_y, p.bbox.max_y, p.displace, whalf, nr, bsize, nrg, merged, &J.y);
  J.thr = p.min_num_points;
  J.n = (int32_t)n;
  g->n = n;
  g->nwin = (int64_t)nc * nr;
  g->ncell = (int64_t)ncg * nrg;
  g->nsub = grid_cells(J);
  J.base[1] = (uint32_t)J.x.width[0] * (uint32_t)J.y.width[0];
  J.base[2] = J.base[1] + (uint32_t)J.x.width[1] * (uint32_t)J.y.width[0];
  J.base[3] = J.base[2] + (uint32_t)J.x.width[0] * (uint32_t)J.y.width[1];
  J.fast = J.x.fast && J.y.fast && (!cells || merged);
  g->bitmap2 = p.overlap > 0.0;
  char* b = static_cast<char*>(scratch);
  size_t o = 0;
  auto take = [&](size_t bytes) -> char* {
    char* q = b ? b + o : nullptr;
    o += up256(bytes);
    return q;
  };
  // cleared
  J.zid = (ulonglong2*)take((size_t)g->nsub * 16);
  J.count = (uint32_t*)take((size_t)g->nsub * 4);
  if (cells && !merged) J.cell_zid = (ulonglong2*)take((size_t)g->ncell * 16);
  const int64_t chunks = ((n + 1 + 31) / 32 + kSeedChunk - 1) / kSeedChunk;
  if (g->bitmap2) {
    J.once = (uint32_t*)take((size_t)(chunks * kSeedChunk) * 4);
    J.twice = (uint32_t*)take((size_t)(chunks * kSeedChunk) * 4);
  }
  J.mark = (uint8_t*)take((size_t)g->ncell);
  g->clear_bytes = o;
  // written by the kernels
  for (int ax = 0; ax < 2; ++ax) {
    GridAxis& a = ax ? J.y : J.x;
    for (int f = 0; f < 4; ++f) a.edge[f] = (int64_t*)take((size_t)(f < 2 ? a.n : a.nc) * 8);
    a.lo = (int32_t*)take((size_t)a.n * 4);
    a.hi = (int32_t*)take((size_t)a.n * 4);
    a.clo = (int32_t*)take((size_t)a.nc * 4);
    a.chi = (int32_t*)take((size_t)a.nc * 4);
  }
  J.occ = (uint32_t*)take(16);
  J.rows = (GridRow*)take((size_t)J.y.nclass * nc * sizeof(GridRow));
  J.cellmin = (uint32_t*)take((size_t)g->ncell * 4);
  g->llp = (uint32_t*)take((size_t)g->nwin * 4);
  g->seeds = (int64_t*)take((size_t)(g->nwin + g->ncell + 1) * 8);
  if (g->bitmap2) {
    g->part = (uint32_t*)take((size_t)chunks * 4);
  } else {
    J.win = (uint32_t*)take((size_t)g->nwin * 4);
    g->s2_bytes = stage2_scratch_bytes(g->nwin);
    g->s2_temp = take(g->s2_bytes);
  }
  if (g->ncell > kOutputCells) {
    g->flags = (uint32_t*)take((size_t)g->ncell * 4);
    g->pos = (uint32_t*)take((size_t)g->ncell * 4);
    g->scan_bytes = scan_temp_bytes(g->ncell);
    g->scan_temp = take(g->scan_bytes);
  }
  g->bytes = o;
  g->base = b;
  return OWM_OK;
}

int grid_prepare(const GridPlan& g, uint32_t* status, cudaStream_t s, int64_t* launches) {
  const int64_t n16 = (int64_t)(g.clear_bytes / 16);
  OWM_LAUNCH("k_grid_prepare", s, k_grid_prepare<<<blocks_for(n16, 152 * 8), 256, 0, s>>>(g.job, (uint4*)g.base, n16, status));
  count_launch(launches);
  OWM_CUDA_TRY(cudaGetLastError());
  return OWM_OK;
}

int grid_fold(const GridPlan& g, const double* rec, int stride, int64_t first, int64_t count, uint32_t* status,
              cudaStream_t s, int64_t* launches) {
  if (count <= 0) return OWM_OK;
  const GridJob& J = g.job;
  const unsigned nb = blocks_for(count, 152 * kFoldBlocks, kFoldBlock);
  auto kernel = J.fast ? (stride == 4 ? k_grid_fold<4, true> : k_grid_fold<3, true>)
                       : (stride == 4 ? k_grid_fold<4, false> : k_grid_fold<3, false>);
  OWM_LAUNCH("k_grid_fold", s, kernel<<<nb, kFoldBlock, 0, s>>>(J, rec, first, count, status));
  count_launch(launches);
  OWM_CUDA_TRY(cudaGetLastError());
  return OWM_OK;
}

int grid_windows(const GridPlan& g, cudaStream_t s, int64_t* launches) {
  const GridJob& J = g.job;
  OWM_LAUNCH("k_grid_rows", s, k_grid_rows<<<blocks_for((int64_t)J.y.nclass * J.x.n, 152 * 32), 256, 0, s>>>(J));
  OWM_LAUNCH("k_grid_windows", s, k_grid_windows<<<blocks_for(g.nwin, 152 * 32), 256, 0, s>>>(J));
  count_launch(launches, 2);
  OWM_CUDA_TRY(cudaGetLastError());
  return OWM_OK;
}

int grid_stage2(const GridPlan& g, const owm_params& p, const double* xy, int xy_stride, uint32_t* d_nllp,
                cudaStream_t s, int64_t* launches) {
  const GridJob& J = g.job;
  if (g.bitmap2) {
    const unsigned chunks = (unsigned)(((g.n + 1 + 31) / 32 + kSeedChunk - 1) / kSeedChunk);
    OWM_LAUNCH("k_grid_seed_count", s, k_grid_seed_count<<<chunks, kSeedBlock, 0, s>>>(J.twice, g.part));
    OWM_LAUNCH("k_grid_seeds", s, k_grid_seeds<<<chunks, kSeedBlock, 0, s>>>(J, g.part, xy, xy_stride, g.llp, d_nllp));
    count_launch(launches, 2);
  } else {
    // overlap 0 keeps every valid minimum, repeated sentinel ids included: by sorting
    const int rc = run_stage2(J.win, g.nwin, g.n, p.overlap, g.llp, d_nllp, g.s2_temp, g.s2_bytes, s, launches);
    if (rc) return rc;
    if (g.ncell) {
      OWM_LAUNCH("k_grid_mark", s, k_grid_mark<<<blocks_for(g.nwin, 152 * 8), 256, 0, s>>>(J, xy, xy_stride, g.llp, d_nllp));
      count_launch(launches);
    }
  }
  OWM_CUDA_TRY(cudaGetLastError());
  return OWM_OK;
}

int grid_stage3(const GridPlan& g, const uint32_t* d_nllp, uint32_t* d_ns3, cudaStream_t s, int64_t* launches) {
  const GridJob& J = g.job;
  if (g.ncell > 0) {
    if (J.cell_zid)
      OWM_LAUNCH("k_grid_cells", s, k_grid_cells_own<<<(unsigned)((g.ncell + 255) / 256), 256, 0, s>>>(J, g.ncell));
    else
      OWM_LAUNCH("k_grid_cells", s, k_grid_cells<<<(unsigned)((g.ncell + 7) / 8), 256, 0, s>>>(J, g.ncell));
    count_launch(launches);
  }
  if (g.ncell <= kOutputCells) {
    OWM_LAUNCH("k_grid_output", s, k_grid_output<<<blocks_for(g.nwin / 4 + g.ncell, 64), kSeedBlock, 0, s>>>(
        J.cellmin, g.ncell, g.llp, d_nllp, g.seeds, d_ns3));
    count_launch(launches);
  } else {
    OWM_LAUNCH("k_grid_flags", s, k_grid_flags<<<blocks_for(g.ncell, 152 * 8), 256, 0, s>>>(J.cellmin, g.ncell, g.flags));
    count_launch(launches);
    OWM_CUDA_TRY(exclusive_scan_u32(g.flags, g.pos, g.ncell, d_ns3, g.scan_temp, g.scan_bytes, s, launches));
    OWM_LAUNCH("k_grid_output", s, k_grid_output_scanned<<<blocks_for(g.nwin + g.ncell, 152 * 8), 256, 0, s>>>(
        J.cellmin, g.pos, g.ncell, g.llp, d_nllp, d_ns3, g.seeds));
    count_launch(launches);
  }
  OWM_CUDA_TRY(cudaGetLastError());
  return OWM_OK;
}

}  // namespace owm

// Host form of the per-axis classification, for tests: the four families'
// edges and, per coordinate, the counts that the fixed-point form gives.
// mode[0]: 1 fixed-point form, [1]: 1 linear, [2]: 1 one parity of classes
// expected empty, [3]: coordinates that the fast form settled.
extern "C" int owm_grid_classify_host(double lo, double hi, double step, int32_t wsize, int32_t n, int32_t bsize, int32_t nc,
                                      const double* p, int64_t np, double* edges, int32_t* counts, int32_t* mode) {
  using namespace owm;
  GridAxis a;
  grid_axis_setup(lo, hi, step, wsize / 2, n, bsize, nc, true, &a);
  mode[0] = a.quick;
  mode[1] = a.linear;
  mode[2] = a.parmask;
  mode[3] = 0;
  double* e = edges;
  for (int f = 0; f < 4; ++f)
    for (int32_t j = 0; j < (f < 2 ? n : nc); ++j) *e++ = dkey_inv(grid_edge(a, f, j));
  for (int64_t i = 0; i < np; ++i) {
    uint64_t b;
    std::memcpy(&b, p + i, 8);
    const int how = grid_counts(a, b, FormulaEdges{&a}, counts + 4 * i);
    if (how == 2) grid_counts_exact(a, b, dkey(p[i]), FormulaEdges{&a}, counts + 4 * i);
    mode[3] += how == 0;
    bool rare = false;
    const int32_t cls = grid_class_fast(a, b, &rare);
    if (a.fast && (rare ? how == 0 : how != 0 || cls != grid_sum(a, counts + 4 * i))) return 1;
  }
  return 0;
}

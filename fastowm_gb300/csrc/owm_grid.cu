// The window-grid path of one cloud (owm_grid.cuh): stage 1
// (optim3_func.cpp:541-561), stage 2 (:610-625) and stage 3 (:627-662) with
// their decisions on exact order keys, in seven launches (small clouds: k_grid_small, the same steps in one):
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
#include <cstddef>
#include <utility>
#include <type_traits>

#include "owm_devutil.cuh"
#include "owm_grid.cuh"

namespace owm {

namespace {

constexpr int kFoldBlock = 256;
constexpr int kFoldBlocks = 6;  // resident fold blocks per SM (40 registers a thread)
// A batch's fold: a block takes a chunk of one tile's points.  Blocks that run
// together take chunks of kTileStripes stretches of the batch: the blocks of one
// tile side by side hit the same few thousand sub-cells (72 M points in 128
// tiles: 1.32 ms in order, 1.18 in 16 stripes, 1.20 in 64, 1.25 in 256).
constexpr int64_t kTileChunk = 4096;
constexpr int kTileStripes = 16;
// Points a full sub-cell from which on the fold reduces a warp's sub-cells one
// after the other (a step for each) instead of all runs of neighbours by a network
// of shuffles: in scan order a warp then meets some five of them.  Fold of 5 M
// points in scan order, one after the other / network: 4 points a sub-cell 87 / 65
// us, 12 69 / 61, 48 54 / 56, 160 49 / 52; 41 M at 48 407 / 416.
constexpr int64_t kFoldDense = 24;

// Start of a kernel of a chain: lets the next one be set up while this one runs
// (its launch latency then overlaps this kernel), and waits until everything
// before this one is done.  Without the launch attribute both do nothing.
// What earlier kernels of the chain write is read by plain loads only: the
// read-only path may be used for data that nothing writes while a kernel
// exists, and it exists before they end.
__device__ __forceinline__ void chain_start() {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Launch of a kernel that starts with chain_start.
template <class... P, class... A>
cudaError_t chain_smem(void (*kernel)(P...), unsigned grid, int block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.dynamicSmemBytes = smem;
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.stream = s;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <class... P, class... A>
cudaError_t chain(void (*kernel)(P...), unsigned grid, int block, cudaStream_t s, A&&... args) {
  return chain_smem(kernel, grid, block, 0, s, std::forward<A>(args)...);
}

__device__ __forceinline__ void stamp(const GridJob& J, int phase) {
  if (J.stamps && blockIdx.x == 0 && threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    J.stamps[phase] = t;
  }
}

// The job that item *k belongs to; *k becomes the item's number within it.
template <bool kMulti>
__device__ __forceinline__ const GridJob& job_at(const GridJob& one, const GridTiles& T, int64_t* k) {
  if (!kMulti) return one;
  const int t = tile_of(T.off, T.n, *k);
  *k -= __ldg(T.off + t);
  return T.jobs[t];
}

// The job of a block that works on one tile of a batch, in shared memory, and
// the tile; *blk becomes the block's number within it.  Every thread of the
// block calls it.  Found per thread instead (a search of log2(tiles) loads one
// after the other, then the job's fields from global memory wherever they are
// used) stage 1's reductions for 72 M points in 128 tiles took 220 us, not 185.
struct BlockJob {
  int tile;
  GridJob job;
};
__device__ __forceinline__ void block_job(const GridTiles& T, BlockJob& S, int64_t* blk) {
  int below = 0;
  for (int j = threadIdx.x; j - (int)threadIdx.x < T.n; j += blockDim.x)
    below += __syncthreads_count(j < T.n && __ldg(T.off + j) <= *blk);
  const int t = below - 1;
  *blk -= __ldg(T.off + t);
  static_assert(sizeof(GridJob) % 16 == 0, "copied in 16-byte words");
  for (int i = threadIdx.x; i < (int)(sizeof(GridJob) / 16); i += blockDim.x)
    reinterpret_cast<uint4*>(&S.job)[i] = __ldg(reinterpret_cast<const uint4*>(T.jobs + t) + i);
  if (threadIdx.x == 0) S.tile = t;
  __syncthreads();
}

// ---- prepare ------------------------------------------------------------------
struct FormulaEdges {
  const GridAxis* a;
  __host__ __device__ __forceinline__ int64_t operator()(int f, int32_t j) const { return grid_edge(*a, f, j); }
};
struct StoredEdges {
  const GridAxis* a;
  __device__ __forceinline__ int64_t operator()(int f, int32_t j) const { return a->edge[f][j]; }
};

// Edge keys and s-range of item i of one axis (windows, then cells), by one
// lane, or by eight neighbouring ones: lanes 0-3 the left edge, 4-7 the right
// one, each counting the edges of one family passed just inside it.  (The
// double-precision sums are a chain of slow operations: one cloud's edges, at
// 10 K points, take 2.1 us by eight lanes an item and 4.7 by one.)
template <int kLanes>
__device__ __forceinline__ void prepare_axis(const GridAxis& a, int32_t i) {
  const bool win = i < a.n;
  const int32_t j = win ? i : i - a.n;
  const int f = win ? kFamL : kFamA;
  auto passed = [&](int q, int64_t key) {
    uint32_t v;
    const bool ok = grid_position(a, (uint64_t)__double_as_longlong(dkey_inv(key)), &v);
    return q < 2 || a.merged ? grid_count_exact(a, q, ok, v, key, FormulaEdges{&a}) : 0;
  };
  int32_t lo = 0, hi = 0;
  int64_t l, r;
  if (kLanes == 8) {
    const int lane = threadIdx.x & 7, q = lane & 3, side = lane >> 2;
    const uint32_t group = 0xFFu << (threadIdx.x & 24);
    const int64_t e = grid_edge(a, f + side, j), other = __shfl_xor_sync(group, e, 4);
    l = side ? other : e;
    r = side ? e : other;
    int32_t c = passed(q, side ? r - 1 : l + 1);
    __syncwarp(group);
    c += __shfl_xor_sync(group, c, 1);
    c += __shfl_xor_sync(group, c, 2);
    lo = c;
    hi = __shfl_xor_sync(group, c, 4);
    if (lane) return;
  } else {
    l = grid_edge(a, f, j);
    r = grid_edge(a, f + 1, j);
    for (int q = 0; q < 4; ++q) lo += passed(q, l + 1);
    for (int q = 0; q < 4; ++q) hi += passed(q, r - 1);
  }
  const_cast<int64_t*>(a.edge[f])[j] = l;
  const_cast<int64_t*>(a.edge[f + 1])[j] = r;
  if (!win && !a.merged) return;
  (win ? a.lo : a.clo)[j] = lo;
  (win ? a.hi : a.chi)[j] = l + 1 <= r - 1 ? hi : -1;  // no double lies between edges that touch: an empty range
}

// Bound by the stores of the clear (20 bytes a sub-cell, 2 bits a point);
// one launch instead of a memset and six small kernels.
template <bool kMulti>
__device__ __forceinline__ void prepare(const GridJob& one, const GridTiles& T, int64_t items, uint4* clear, int64_t nclear,
                                        int64_t t, int64_t nt) {
  if (one.stamps && blockIdx.x == 0 && threadIdx.x == 0) one.stamps[1] = one.stamps[2] = one.stamps[3] = 0;
  stamp(one, 0);
  const uint4 z = make_uint4(0, 0, 0, 0);  // the stores drain under the edges' arithmetic
  for (int64_t i = t; i < nclear; i += nt) clear[i] = z;
  constexpr int kLanes = kMulti ? 1 : 8;  // 128 tiles' items fill the chip by themselves (68 us; 72 by eight lanes)
  for (int64_t i = t; i < kLanes * items; i += nt) {  // nt: whole warps
    int64_t k = i / kLanes;
    const GridJob& J = job_at<kMulti>(one, T, &k);
    const int32_t nx = J.x.n + J.x.nc, ny = J.y.n + J.y.nc;
    if (k < nx) {
      prepare_axis<kLanes>(J.x, (int32_t)k);
    } else if (k < nx + ny) {
      prepare_axis<kLanes>(J.y, (int32_t)k - nx);
    } else if (t % kLanes == 0) {
      const int q = (int)(k - nx - ny);
      J.occ[q] = (q & 1) == 0;  // the other parity: when a point says so
    }
  }
}
template <bool kMulti>
__global__ void __launch_bounds__(256) k_grid_prepare(const __grid_constant__ GridJob one, GridTiles T, int64_t items,
                                                      uint4* clear, int64_t nclear, uint32_t* status) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0) *status = 0;
  prepare<kMulti>(one, T, items, clear, nclear, t, (int64_t)gridDim.x * blockDim.x);
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

// Point i as raw bits, and its inverted id; every point is read once.
template <int kStride>
__device__ __forceinline__ void load_raw(const GridPoints& pts, uint32_t i, uint64_t& x, uint64_t& y, uint64_t& z,
                                         uint32_t& nid) {
  if (kStride == 4) {
    asm("ld.global.nc.L1::no_allocate.L2::evict_first.v4.b64 {%0, %1, %2, _}, [%3];"
        : "=l"(x), "=l"(y), "=l"(z)
        : "l"(pts.rec + 4 * (uint64_t)i));
    nid = ~(i + 1);
  } else if (kStride == 3) {
    const uint64_t* p = reinterpret_cast<const uint64_t*>(pts.rec) + 3 * (uint64_t)i;
    x = __ldg(p);
    y = __ldg(p + 1);
    z = __ldg(p + 2);
    nid = ~(i + 1);
  } else {
    x = (uint64_t)__double_as_longlong(dkey_inv(__ldg(pts.xk + i)));
    y = (uint64_t)__double_as_longlong(dkey_inv(__ldg(pts.yk + i)));
    z = (uint64_t)__double_as_longlong(dkey_inv(__ldg(pts.zk + i)));
    nid = ~__ldg(pts.id + i);
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
constexpr uint32_t kCrowded = 8;  // of a lane of the fold: shared its sub-cell with lanes further off

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

// Points [b, e) of a cloud or tile into their sub-cells, 32 at a time (e a
// multiple of 32 above b).  kFast: both axes have the
// fast form; a point near an edge is settled by the edges its places end at,
// and one outside the box, or with z zero or not finite, takes the full form in
// a call.
//
// Bound by the L2 requests of points in no order (a read and an add each): 100 M
// points into 0.9 M sub-cells take 0.97 ms (32 bytes a point: 3.3 TB/s), a bare
// kernel that does just those two requests 0.87.  In scan order it is bound by
// latency and instructions (issue 51 %).  What cost more before:
// - the order of the work: a warp takes a stretch of neighbouring points, so
//   that scan lines side by side are not folded at the same time (40 M points in
//   scan order at 3 a square metre: 1.28 -> 0.53 ms);
// - instructions: 144 per 32 points instead of 284 (0.53 -> 0.40 ms there);
// - lanes of one sub-cell reduced on 96 bits where the top half of their heights
//   tells them apart (0.45 -> 0.41 ms there, in whole centimetres);
// - an add for each run of neighbours where the lanes of one sub-cell lie apart:
//   its adds queue in L2 (a cloud crowded in a few places, in no order: 20 M
//   points, half of them within a metre, 3.4 -> 0.6 to 1.0 ms; 1 / r^2 around one
//   place 1.7 -> 1.0).  Such lanes are found where neighbours share a sub-cell,
//   and looked for in every group of 32 once a warp has met some;
// - points on edges (whole centimetres: 1 in 100): two loads side by side in
//   place of a call (20 M in no order 0.37 -> 0.24 ms, in scan order 0.28 -> 0.23).
// One point a thread at 48 warps an SM: two at 40 took 1.05 ms for the 100 M,
// four at 32 1.05, and 0.46 for the scan.  A single add whose result carries a
// filter for the minimum took 1.40.
// The fast form's constants where the fold finds them: the kernel's parameters,
// or (a batch) the tile's job in shared memory, read anew for each group of
// points in 16-byte words (kept in registers they would halve the warps).
struct ParamAxes {
  const GridJob* J;
  __device__ __forceinline__ const GridAxis& x() const { return J->x; }
  __device__ __forceinline__ const GridAxis& y() const { return J->y; }
};
struct SharedAxes {
  const GridJob* J;
  static __device__ __forceinline__ GridFastAxis load(const GridAxis* a) {
    GridFastAxis f;
    uint4 w[5];
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(a);
#pragma unroll
    for (int k = 0; k < 5; ++k)
      asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(w[k].x), "=r"(w[k].y), "=r"(w[k].z), "=r"(w[k].w)
                   : "r"(at + 16 * k));
    memcpy(&f, w, sizeof(f));
    return f;
  }
  __device__ __forceinline__ GridFastAxis x() const { return load(&J->x); }
  __device__ __forceinline__ GridFastAxis y() const { return load(&J->y); }
};

// A point's sub-cell and z on axes with the fast form.
template <bool kPaired, class Axes>
__device__ __forceinline__ void fast_cell(const GridJob& J, Axes axes, uint64_t x, uint64_t y, uint64_t z, uint32_t& cell,
                                          unsigned long long& w, uint32_t& flags) {
  int32_t tx[4], ty[4];
  uint32_t hx, hy, other;
  const auto& ax = axes.x();
  int32_t sx = grid_class_fast<kPaired>(ax, x, &hx, tx);
  other = (sx ^ ax.par) & ax.parmask;
  const uint32_t ix = (uint32_t)(sx >> ax.parmask);
  const auto& ay = axes.y();
  int32_t sy = grid_class_fast<kPaired>(ay, y, &hy, ty);
  other |= (sy ^ ay.par) & ay.parmask;
  cell = (uint32_t)(sy >> ay.parmask) * (uint32_t)J.x.width[0] + ix;
  w = z ^ (~(uint64_t)((int64_t)z >> 63) & 0x7FFFFFFFFFFFFFFFull);
  const bool odd_z = ((uint32_t)(z >> 32) << 1) - 1u >= 0xFFDFFFFFu;  // zero or not finite
  if (odd_z | (other | hx | hy)) {
    if (odd_z | ((hx | hy) & kGridOutside)) {
      const PointCell p = point_cell_call(J, x, y, z);
      cell = p.cell;
      w = p.w;
      flags |= p.flags;
    } else {
      if (hx) sx = grid_settle_fast(J.x, (int64_t)x, hx, tx, StoredEdges{&J.x}, sx);
      if (hy) sy = grid_settle_fast(J.y, (int64_t)y, hy, ty, StoredEdges{&J.y}, sy);
      cell = grid_cell(J, sx, sy);
      flags |= (((sx ^ J.x.par) & J.x.parmask) ? kPointOtherX : 0u) | (((sy ^ J.y.par) & J.y.parmask) ? kPointOtherY : 0u);
    }
  }
}

template <int kStride, int kFast, bool kSparse, class Axes>
__device__ __forceinline__ void fold_stretch(const GridJob& J, Axes axes, const GridPoints& pts, uint32_t b, uint32_t e,
                                             uint32_t& flags) {
  const int lane = threadIdx.x & 31;
  for (; b < e; b += 32) {
    // lanes past the end take the last point again, and are not counted
    const int32_t left = (int32_t)min(32u, (uint32_t)J.n - b);
    const uint32_t i = b + (uint32_t)min(lane, left - 1);
    uint64_t x, y, z;
    uint32_t cell, nid;
    load_raw<kStride>(pts, i, x, y, z, nid);
    unsigned long long w;
    if (kFast) {
      fast_cell<kFast == 2>(J, axes, x, y, z, cell, w, flags);
    } else {
      const PointCell p = point_cell(J, x, y, z);
      cell = p.cell;
      w = p.w;
      flags |= p.flags;
      if (J.cell_zid) raise_own_cells(J, x, y, w, nid);
    }
    const ulonglong2 cur = load_zid(J.zid + cell);
    // neighbouring lanes in one sub-cell (a cloud in scan order)
    const uint32_t before = __shfl_up_sync(0xffffffffu, cell, 1);
    const uint32_t heads = __ballot_sync(0xffffffffu, before != cell) | 1u;
    if (heads == 0xFFFFFFFFu && !__any_sync(0xffffffffu, flags & kCrowded)) {  // none (a lane past the end would repeat its neighbour)
      atomicAdd(J.count + grid_count_slot(J, cell), 1u);
      if (w >= cur.x) raise_zid(J.zid + cell, cur, w, nid);
      continue;
    }
    const uint32_t group = __match_any_sync(0xffffffffu, cell);
    if ((group & (0u - group)) == 1u << lane)
      atomicAdd(J.count + grid_count_slot(J, cell), (uint32_t)__popc(group & (0xFFFFFFFFu >> (32 - left))));
    const uint32_t from = group >> lane;
    if (from & (from + 1)) flags |= kCrowded;
    if (!__any_sync(0xffffffffu, w >= cur.x)) continue;
    // the lane with the highest top half of w in its group, or in its run of
    // neighbours (kFoldDense), raises the entry
    const uint32_t top = (uint32_t)(w >> 32);
    bool raise = w >= cur.x;
    if (!kSparse) {
      const uint32_t most = __reduce_max_sync(group, top);  // by every lane, raising or not
      raise = raise && most == top;
      const uint32_t several = __ballot_sync(0xffffffffu, raise) & group;
      if (__any_sync(0xffffffffu, (several & (several - 1)) != 0)) {
        raise = raise && zid_above(w, nid, cur);
        if (__any_sync(0xffffffffu, raise)) {  // none on flat ground: its ids rise
          const uint32_t low = __reduce_max_sync(group, raise ? (uint32_t)w : 0u);
          raise = raise && (uint32_t)w == low;
          const uint32_t best = __reduce_max_sync(group, raise ? nid : 0u);
          raise = raise && nid == best;
        }
      }
    } else {
      const uint32_t after = heads & (0xFFFFFFFEu << lane);
      const int end = after ? __ffs(after) - 1 : 32, start = 31 - __clz(heads & (0xFFFFFFFFu >> (31 - lane)));
      uint32_t most = top;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {  // the run's highest, to its head and from there to all
        const uint32_t other = __shfl_down_sync(0xffffffffu, most, o);
        if (lane + o < end) most = max(most, other);
      }
      most = __shfl_sync(0xffffffffu, most, start);
      raise = raise && most == top;
      const uint32_t several = __ballot_sync(0xffffffffu, raise) & (0xFFFFFFFFu << start) & (0xFFFFFFFFu >> (32 - end));
      if (__any_sync(0xffffffffu, (several & (several - 1)) != 0)) {
        raise = raise && zid_above(w, nid, cur);
        if (__any_sync(0xffffffffu, raise)) {
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {  // the run's minimum, to its head
            const unsigned long long ow = __shfl_down_sync(0xffffffffu, w, o);
            const uint32_t on = __shfl_down_sync(0xffffffffu, nid, o);
            if (lane + o < end && (ow > w || (ow == w && on > nid))) {
              w = ow;
              nid = on;
            }
          }
          raise = (heads >> lane) & 1u;
        }
      }
    }
    if (raise) raise_zid(J.zid + cell, cur, w, nid);
  }
}

// What a warp found out, stored unless another one did: stores to the one word
// queue.  A store per point cost 0.4 ms on 40 M points in whole centimetres, and
// one per warp 0.3 ms on 5 M points in no order and in multiples of 2 m (384 -> 78
// us).
__device__ __forceinline__ void fold_flags(const GridJob& J, uint32_t flags, uint32_t* __restrict__ status) {
  flags = __reduce_or_sync(0xffffffffu, flags);
  if ((threadIdx.x & 31) == 0 && flags) {
    if (flags & kPointNonFinite) atomicOr(status, kStatusNonFinite);
    volatile uint32_t* occ = J.occ;
    if ((flags & kPointOtherX) && !occ[1]) occ[1] = 1;
    if ((flags & kPointOtherY) && !occ[3]) occ[3] = 1;
  }
}

template <int kStride, int kFast, bool kSparse>
__global__ void __launch_bounds__(kFoldBlock, kFoldBlocks)
    k_grid_fold(const __grid_constant__ GridJob J, const __grid_constant__ GridPoints pts, uint32_t* __restrict__ status) {
  chain_start();
  const int64_t nwarps = ((int64_t)gridDim.x * kFoldBlock) >> 5;
  uint32_t flags = 0;
  int64_t t0, t1;
  chunk_tiles(((int64_t)J.n + 31) / 32, nwarps, ((int64_t)blockIdx.x * kFoldBlock + threadIdx.x) >> 5, &t0, &t1);
  fold_stretch<kStride, kFast, kSparse>(J, ParamAxes{&J}, pts, (uint32_t)(t0 * 32), (uint32_t)(t1 * 32), flags);
  fold_flags(J, flags, status);
}

// The fold where points are many and sub-cells few (wide windows, dense points):
// there the adds and swaps of one address queue in L2.  Each block folds a
// stretch of the points into a table of its own in shared memory, kFewPer points
// a thread at a time, and then raises the job's entries once per sub-cell.  An
// entry's id belongs to the height in tag: a lower point in a later group resets
// it first.  Bound by latency up to about 0.6 M points (one group a block), then
// by the shared atomics: 2 M points on 2401 sub-cells 99 -> 31 us, 20 M on 3249
// 872 -> 176.
constexpr int kFewBlock = 1024, kFewPer = 4;
constexpr size_t few_bytes(int64_t nsub) { return 24 * (size_t)nsub; }
template <int kStride>
__global__ void __launch_bounds__(kFewBlock)
    k_grid_fold_few(const __grid_constant__ GridJob J, const __grid_constant__ GridPoints pts, uint32_t nsub, uint32_t* status) {
  extern __shared__ __align__(256) char mem[];
  unsigned long long* top = reinterpret_cast<unsigned long long*>(mem);
  unsigned long long* tag = top + nsub;
  uint32_t* id = reinterpret_cast<uint32_t*>(tag + nsub);
  uint32_t* count = id + nsub;
  chain_start();
  const uint32_t t = threadIdx.x;
  for (uint32_t c = t; c < nsub; c += kFewBlock) {
    top[c] = tag[c] = 0;
    id[c] = count[c] = 0;
  }
  __syncthreads();
  const uint32_t n = (uint32_t)J.n, per = (n + gridDim.x - 1) / gridDim.x;
  const uint32_t first = min(n, blockIdx.x * per), last = min(n, first + per);
  uint32_t flags = 0;
  for (uint32_t b = first; b < last; b += kFewBlock * kFewPer) {
    uint64_t x[kFewPer], y[kFewPer], w[kFewPer];
    uint32_t nid[kFewPer], cell[kFewPer];
    const uint32_t left = last - b;
#pragma unroll
    for (int k = 0; k < kFewPer; ++k)
      if (k * kFewBlock + t < left) load_raw<kStride>(pts, b + k * kFewBlock + t, x[k], y[k], w[k], nid[k]);
#pragma unroll
    for (int k = 0; k < kFewPer; ++k)
      if (k * kFewBlock + t < left) {
        if (J.fast == 2) {
          unsigned long long v;
          fast_cell<true>(J, ParamAxes{&J}, x[k], y[k], w[k], cell[k], v, flags);
          w[k] = v;
        } else if (J.fast) {
          unsigned long long v;
          fast_cell<false>(J, ParamAxes{&J}, x[k], y[k], w[k], cell[k], v, flags);
          w[k] = v;
        } else {
          const PointCell p = point_cell_call(J, x[k], y[k], w[k]);
          cell[k] = p.cell;
          w[k] = p.w;
          flags |= p.flags;
          if (J.cell_zid) raise_own_cells(J, x[k], y[k], p.w, nid[k]);
        }
        atomicAdd(count + cell[k], 1u);
        if (w[k] > top[cell[k]]) atomicMax(top + cell[k], (unsigned long long)w[k]);
      }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kFewPer; ++k)
      if (k * kFewBlock + t < left && w[k] == top[cell[k]] && tag[cell[k]] != w[k]) {
        tag[cell[k]] = w[k];
        id[cell[k]] = 0;
      }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kFewPer; ++k)
      if (k * kFewBlock + t < left && w[k] == top[cell[k]]) atomicMax(id + cell[k], nid[k]);
    __syncthreads();
  }
  fold_flags(J, flags, status);
  // blocks start at different sub-cells
  const uint32_t start = (uint32_t)((uint64_t)nsub * blockIdx.x / gridDim.x);
  for (uint32_t i = t; i < nsub; i += kFewBlock) {
    const uint32_t c = i + start < nsub ? i + start : i + start - nsub;
    if (!count[c]) continue;
    atomicAdd(J.count + grid_count_slot(J, c), count[c]);
    raise_zid(J.zid + c, load_zid(J.zid + c), top[c], id[c]);
  }
}

// A batch: block b takes one chunk of its tile's points, with the tile's job in
// shared memory.
__global__ void __launch_bounds__(kFoldBlock, kFoldBlocks)
    k_grid_fold_tiles(GridTiles T, int32_t chunk, uint32_t* __restrict__ status) {
  __shared__ __align__(16) BlockJob S;
  int64_t blk = (int64_t)(blockIdx.x % kTileStripes) * (gridDim.x / kTileStripes) + blockIdx.x / kTileStripes;
  if (blk >= __ldg(T.off + T.n)) return;
  block_job(T, S, &blk);
  const GridJob& J = S.job;
  const int64_t c0 = blk * (int64_t)chunk;
  const int64_t n = min((int64_t)chunk, J.n - c0);  // points of this block
  GridPoints pts;
  pts.rec = J.rec;
  uint32_t flags = 0;
  int64_t t0, t1;
  chunk_tiles((n + 31) / 32, kFoldBlock / 32, threadIdx.x >> 5, &t0, &t1);
  const uint32_t b = (uint32_t)(c0 + t0 * 32), e = (uint32_t)(c0 + t1 * 32);
  if (J.fast == 2)
    J.sparse ? fold_stretch<3, 2, true>(J, SharedAxes{&J}, pts, b, e, flags) : fold_stretch<3, 2, false>(J, SharedAxes{&J}, pts, b, e, flags);
  else if (J.fast)
    J.sparse ? fold_stretch<3, 1, true>(J, SharedAxes{&J}, pts, b, e, flags) : fold_stretch<3, 1, false>(J, SharedAxes{&J}, pts, b, e, flags);
  else
    fold_stretch<3, 0, true>(J, SharedAxes{&J}, pts, b, e, flags);
  fold_flags(J, flags, status);
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

// First and last stored index of the classes lo..hi of the main (q = 0) or the
// other parity; false when there are none or they hold no point.
__device__ __forceinline__ bool parity_range(const GridAxis& a, const uint32_t* occ, int q, int32_t lo, int32_t hi,
                                             int32_t* i0, int32_t* i1) {
  if (!occ[q]) return false;
  if (a.parmask) {
    const int32_t par = a.par ^ q;
    lo += (lo ^ par) & 1;
    hi -= (hi ^ par) & 1;
  }
  *i0 = lo >> a.parmask;
  *i1 = hi >> a.parmask;
  return lo <= hi;
}

// A thread per sub-cell row and window column.  A batch's block takes rows of
// one tile.
__device__ __forceinline__ void rows_of(const GridJob& J, int64_t item) {
  if (item >= (int64_t)J.y.nclass * J.x.n) return;
  const uint32_t k = (uint32_t)item;  // below 2^32, as the sub-cells are
  const int32_t r = (int32_t)(k / (uint32_t)J.x.n), ii = (int32_t)(k % (uint32_t)J.x.n);
  const int qy = r >= J.y.width[0];
  if (!J.occ[2 + qy]) return;
  const int32_t iy = r - (qy ? J.y.width[0] : 0), lo = J.x.lo[ii], hi = J.x.hi[ii];
  Best m;
  for (int q = 0; q < 2; ++q) {
    int32_t i0, i1;
    if (!parity_range(J.x, J.occ, q, lo, hi, &i0, &i1)) continue;
    const int64_t at = J.base[2 * qy + q] + (int64_t)iy * J.x.width[q];
    for (int64_t c = at + i0; c <= at + i1; ++c) {
      const ulonglong2 e = J.zid[c];
      m.count += J.count[grid_count_slot(J, (uint32_t)c)];
      m.take(e.x, (uint32_t)e.y);
    }
  }
  GridRow o;
  o.w = m.w;
  o.nid = m.nid;
  o.count = m.count;
  J.rows[k] = o;
}

template <bool kMulti>
__global__ void __launch_bounds__(256) k_grid_rows(const __grid_constant__ GridJob one, GridTiles T) {
  chain_start();
  stamp(one, 1);
  int64_t blk = blockIdx.x;
  if (kMulti) {
    __shared__ __align__(16) BlockJob S;
    block_job(T, S, &blk);
    rows_of(S.job, blk * 256 + threadIdx.x);
  } else {
    rows_of(one, blk * 256 + threadIdx.x);
  }
}

__device__ __forceinline__ void window_of(const GridJob& J, int64_t item) {
  if (item >= (int64_t)J.y.n * J.x.n) return;
  // the search starts from the reference's sentinel point 0 {0, 0, DBL_MAX}
  const unsigned long long sentinel = ~((unsigned long long)kZSentinel ^ 0x8000000000000000ull);
  const uint32_t k = (uint32_t)item;
  const int32_t jj = (int32_t)(k / (uint32_t)J.x.n), ii = (int32_t)(k % (uint32_t)J.x.n);
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
    s2_mark_id<false>(J.once, J.twice, (uint32_t)J.n, id);
}

template <bool kMulti>
__global__ void __launch_bounds__(256) k_grid_windows(const __grid_constant__ GridJob one, GridTiles T) {
  chain_start();
  int64_t blk = blockIdx.x;
  if (kMulti) {
    __shared__ __align__(16) BlockJob S;
    block_job(T, S, &blk);
    window_of(S.job, blk * 256 + threadIdx.x);
  } else {
    window_of(one, blk * 256 + threadIdx.x);
  }
}

// ---- stage 2 ------------------------------------------------------------------
constexpr int kSeedBlock = 256;
constexpr int64_t kSeedChunk = 4 * (int64_t)kSeedBlock;  // bitmap words a block takes

template <int kBlock = kSeedBlock>
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* total) {
  __shared__ uint32_t ws[kBlock / 32];
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
  uint32_t before = 0;
  if (kBlock > 256) {
    uint32_t sum = ws[lane % (kBlock / 32)];
#pragma unroll
    for (int o = 1; o < kBlock / 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += t;
    }
    *total = __shfl_sync(0xffffffffu, sum, kBlock / 32 - 1);
    if (w) before = __shfl_sync(0xffffffffu, sum, w - 1);
  } else {
    uint32_t all = 0;
#pragma unroll
    for (int q = 0; q < kBlock / 32; ++q) {
      const uint32_t x = ws[q];
      before += q < w ? x : 0u;
      all += x;
    }
    *total = all;
  }
  return before + inc - v;
}

__global__ void __launch_bounds__(kSeedBlock) k_grid_seed_count(const uint32_t* bm, uint32_t* __restrict__ part) {
  chain_start();
  const uint4 q = reinterpret_cast<const uint4*>(bm)[(int64_t)blockIdx.x * kSeedBlock + threadIdx.x];
  uint32_t total;
  block_exclusive((uint32_t)(__popc(q.x) + __popc(q.y) + __popc(q.z) + __popc(q.w)), &total);
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
// all chunks before it (whose counts, or words when part is null, it adds up)
// and marks their cells.
// A batch: tile by tile; nllp[t] is tile t's first LLP, nllp[T.n] their number.
// The ids are listed first and then taken a thread each: the points' loads and
// the marks of a chunk are in flight together (in the loop over a thread's
// words they came one after the other: 24 us for 100 M points, now 18; 87 for 72
// M in 128 tiles, now 50).
template <bool kMulti, int kBlock = kSeedBlock>
__device__ __forceinline__ void write_seeds(const GridJob& J, const GridTiles& T, int tile, int64_t chunk, uint32_t blocks, const uint32_t* part,
                                            const double* __restrict__ xy, int stride, uint32_t* llp, uint32_t* nllp) {
  uint32_t before = 0, total;
  if (part) {
    for (uint32_t q = threadIdx.x; q < blockIdx.x; q += kBlock) before += part[q];
  } else {  // few chunks: their words themselves
    const uint4* w = reinterpret_cast<const uint4*>(J.twice);
    const uint32_t words = blockIdx.x * (uint32_t)(kSeedChunk / 4);
    for (uint32_t q = threadIdx.x; q < words; q += kBlock) {
      const uint4 v = w[q];
      before += (uint32_t)(__popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w));
    }
  }
  block_exclusive<kBlock>(before, &before);
  constexpr int kWords = (int)(kSeedChunk / kBlock);  // of a thread
  static_assert(kWords == 4 || kWords == 1, "one load");
  const int64_t w0 = chunk * kSeedChunk + (int64_t)threadIdx.x * kWords;
  const uint4 q = kWords == 4 ? *reinterpret_cast<const uint4*>(J.twice + w0) : make_uint4(J.twice[w0], 0, 0, 0);
  const uint32_t word[4] = {q.x, q.y, q.z, q.w};
  uint32_t at = before + block_exclusive<kBlock>((uint32_t)(__popc(q.x) + __popc(q.y) + __popc(q.z) + __popc(q.w)), &total);
  if (threadIdx.x == 0) {
    if (kMulti && chunk == 0) nllp[tile] = before;
    if (blockIdx.x == blocks - 1) nllp[kMulti ? T.n : 0] = before + total;
  }
#pragma unroll
  for (int k = 0; k < kWords; ++k) {
    uint32_t b = word[k];
    while (b) {
      llp[at++] = (uint32_t)((w0 + k) * 32) + (uint32_t)(__ffs(b) - 1);
      b &= b - 1;
    }
  }
  if (!J.x.nc) return;
  __syncthreads();  // the whole block's list
  for (uint32_t k = before + threadIdx.x; k < before + total; k += kBlock)
    mark_cells(J, kMulti ? J.rec : xy, kMulti ? 3 : stride, llp[k]);
}

template <bool kMulti>
__global__ void __launch_bounds__(kSeedBlock) k_grid_seeds(const __grid_constant__ GridJob one, GridTiles T,
                                                           const uint32_t* part, const double* __restrict__ xy, int stride,
                                                           uint32_t* llp, uint32_t* nllp) {
  chain_start();
  stamp(one, 2);
  int64_t chunk = blockIdx.x;
  if (kMulti) {
    __shared__ __align__(16) BlockJob S;
    block_job(T, S, &chunk);
    write_seeds<true>(S.job, T, S.tile, chunk, gridDim.x, part, xy, stride, llp, nllp);
  } else {
    write_seeds<false>(one, T, 0, chunk, gridDim.x, part, xy, stride, llp, nllp);
  }
}

// The cells of LLPs that another kernel listed.
__global__ void __launch_bounds__(256) k_grid_mark(const __grid_constant__ GridJob J, const double* __restrict__ xy, int stride,
                                                   const uint32_t* __restrict__ llp, const uint32_t* __restrict__ nllp) {
  stamp(J, 2);
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

// One warp per cell: the (z, id)-min of its rectangle of sub-cells, or its own
// entry.
__device__ __forceinline__ void cell_of(const GridJob& J, int64_t c) {
  const int lane = threadIdx.x & 31;
  const int32_t ci = (int32_t)(c % J.x.nc), cj = (int32_t)(c / J.x.nc);
  Best m;
  if (J.cell_zid) {
    const ulonglong2 e = J.cell_zid[c];
    if (!J.mark[c]) m.take(e.x, (uint32_t)e.y);
  } else if (!J.mark[c]) {
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

template <bool kMulti>
__global__ void __launch_bounds__(256) k_grid_cells(const __grid_constant__ GridJob one, GridTiles T, int64_t total) {
  chain_start();
  stamp(one, 3);
  int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= total) return;
  const GridJob& J = job_at<kMulti>(one, T, &c);
  cell_of(J, c);
}

// The result's words (ResultBuffer), by one thread once the counts are known.
__device__ __forceinline__ void write_words(const GridJob& J, const GridResult& R, uint32_t nllp, uint32_t ns3) {
  *R.ns3 = ns3;
  R.words[kResultStatus] = *R.status;
  R.words[kResultLlp] = nllp;
  R.words[kResultS3] = ns3;
  unsigned long long* to = reinterpret_cast<unsigned long long*>(R.words + 16);
  unsigned long long t = 0;
  for (int k = 0; k < kGridStamps - 1; ++k) to[k] = t = J.stamps[k] ? J.stamps[k] : t;  // a phase without a kernel: 0 long
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  to[kGridStamps - 1] = t;
  R.words[8] = 1;
}

// seeds = the valid entries of cellmin in order, then the LLPs.  Every block
// counts all cells (at most kOutputCells) for the total and its own start.
constexpr int64_t kOutputCells = 32768;
template <int kBlock>
__device__ __forceinline__ void write_output(const GridJob& J, int64_t ncell, const uint32_t* llp, const GridResult& R, int64_t blk,
                                             int64_t blocks) {
  const int64_t per = (ncell + blocks - 1) / blocks;
  const int64_t b0 = per * blk, b1 = min(b0 + per, ncell);
  uint32_t before = 0, all = 0;
  for (int64_t i = threadIdx.x; i < ncell; i += kBlock) {
    const uint32_t v = J.cellmin[i] != kNone ? 1u : 0u;
    all += v;
    if (i < b0) before += v;
  }
  block_exclusive<kBlock>(before, &before);
  block_exclusive<kBlock>(all, &all);
  uint32_t at = before;
  for (int64_t t = b0; t < b1; t += kBlock) {
    const uint32_t v = t + threadIdx.x < b1 ? J.cellmin[t + threadIdx.x] : kNone;
    uint32_t got;
    const uint32_t p = block_exclusive<kBlock>(v != kNone ? 1u : 0u, &got);
    if (v != kNone) R.seeds[at + p] = v;
    at += got;
  }
  const uint32_t n = *R.nllp;
  for (uint32_t k = (uint32_t)blk * kBlock + threadIdx.x; k < n; k += (uint32_t)blocks * kBlock) R.seeds[all + k] = llp[k];
  if (blk == 0 && threadIdx.x == 0) write_words(J, R, n, all);
}

__global__ void __launch_bounds__(kSeedBlock) k_grid_output(const __grid_constant__ GridJob J, int64_t ncell, const uint32_t* llp,
                                                            GridResult R) {
  chain_start();
  write_output<kSeedBlock>(J, ncell, llp, R, blockIdx.x, gridDim.x);
}

// ---- small clouds: all of it in one launch -----------------------------------------
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// This block's address of p (in shared memory) in the block of that rank.
template <class T>
__device__ __forceinline__ T* in_block(T* p, int rank) {
  T* q;
  asm("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"(p), "r"(rank));
  return q;
}

constexpr int kSmallCluster = 8, kSmallBlock = 1024, kSmallPer = 4;
// Points: at most kSmallPer a thread, and ids in one chunk of the bitmaps.
constexpr int64_t kSmallPoints = (int64_t)kSmallCluster * kSmallBlock * kSmallPer - 1;
static_assert((kSmallPoints + 1 + 31) / 32 <= kSeedChunk, "one chunk");

// The 8-byte words of a GridJob that are addresses of its tables.
struct JobTables {
  uint64_t m[2];
};
constexpr JobTables job_tables() {
  JobTables w{};
  constexpr size_t x = offsetof(GridJob, x), y = offsetof(GridJob, y);
  const size_t at[] = {offsetof(GridJob, zid), offsetof(GridJob, count), offsetof(GridJob, rows), offsetof(GridJob, occ),
                       offsetof(GridJob, mark), offsetof(GridJob, cellmin), offsetof(GridJob, once), offsetof(GridJob, twice)};
  for (size_t a : at) w.m[a / 512] |= 1ull << (a / 8 % 64);
  for (size_t axis : {x, y}) {
    for (size_t k = 0; k < 4; ++k) {
      const size_t a = axis + offsetof(GridAxis, edge) + 8 * k;
      w.m[a / 512] |= 1ull << (a / 8 % 64);
    }
    for (size_t f : {offsetof(GridAxis, lo), offsetof(GridAxis, hi), offsetof(GridAxis, clo), offsetof(GridAxis, chi)})
      w.m[(axis + f) / 512] |= 1ull << ((axis + f) / 8 % 64);
  }
  return w;
}
constexpr uint64_t kJobTables0 = job_tables().m[0], kJobTables1 = job_tables().m[1];
static_assert(sizeof(GridJob) <= 1024 && sizeof(GridJob) % 8 == 0, "two words of 64 bits");

// The whole path of a small cloud by one cluster, with every table of the plan
// in shared memory: each block folds an eighth of the points into tables of its
// own (minimum of z first, then of the ids that have it), the blocks merge a
// slice of the sub-cells each into the first one's, and that one does the rest.
// Bound by latency, about 2 us each for the edges, the fold, the merge, the
// reductions, the seeds and the output.  10 K points take 34 us a call and as a
// chain of seven kernels, which meet in L2, 46 (the launches hide behind the
// kernels: the same steps in one launch on global tables took 43).
// base: where the plan's tables would lie.
template <int kStride>
__global__ void __cluster_dims__(kSmallCluster) __launch_bounds__(kSmallBlock)
    k_grid_small(const __grid_constant__ GridJob G, const __grid_constant__ GridPoints pts, const char* base, int64_t items,
                 int64_t nclear, uint32_t nsub, const double* __restrict__ xy, int xy_stride, int32_t ncell,
                 int64_t llp_at, const __grid_constant__ GridResult R) {
  extern __shared__ __align__(256) char mem[];
  __shared__ __align__(16) GridJob J;
  __shared__ uint32_t words[4];
  __shared__ unsigned long long stamps[kGridStamps];
  const int t = threadIdx.x, rank = blockIdx.x;
  const int64_t delta = (int64_t)mem - (int64_t)base;  // whole numbers: an address made from a parameter's is taken for global memory
  uint32_t* llp = reinterpret_cast<uint32_t*>(mem + llp_at);
  if (t < (int)(sizeof(GridJob) / 8)) {  // the job, its tables' addresses moved here
    int64_t v = reinterpret_cast<const int64_t*>(&G)[t];
    if ((((t < 64 ? kJobTables0 : kJobTables1) >> (t & 63)) & 1) && v) v += delta;
    if (t == (int)(offsetof(GridJob, stamps) / 8)) v = (int64_t)stamps;
    reinterpret_cast<int64_t*>(&J)[t] = v;
  }
  GridResult out = R;  // the words that it reads again itself
  out.status = &words[0];
  out.nllp = &words[1];
  out.ns3 = &words[2];
  if (t < 4) words[t] = 0;
  const int per = (G.n + kSmallCluster - 1) / kSmallCluster, first = rank * per + t, last = min(G.n, (rank + 1) * per);
  // the points' loads go out before the tables are ready
  uint64_t x[kSmallPer], y[kSmallPer], z[kSmallPer];
  uint32_t nid[kSmallPer], cell[kSmallPer];
#pragma unroll
  for (int k = 0; k < kSmallPer; ++k) {
    const int i = first + k * kSmallBlock;
    if (i < last) load_raw<kStride>(pts, i, x[k], y[k], z[k], nid[k]);
  }
  __syncthreads();
  prepare<false>(J, GridTiles{}, items, reinterpret_cast<uint4*>(mem), nclear, t, kSmallBlock);
  __syncthreads();
  uint32_t flags = 0;
#pragma unroll
  for (int k = 0; k < kSmallPer; ++k) {
    if (first + k * kSmallBlock >= last) break;
    if (J.fast == 2) {
      unsigned long long w;
      fast_cell<true>(J, ParamAxes{&J}, x[k], y[k], z[k], cell[k], w, flags);
      z[k] = w;
    } else {
      const PointCell p = point_cell_call(J, x[k], y[k], z[k]);
      cell[k] = p.cell;
      z[k] = p.w;
      flags |= p.flags;
    }
    atomicAdd(J.count + grid_count_slot(J, cell[k]), 1u);
    atomicMax(&J.zid[cell[k]].x, (unsigned long long)z[k]);
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kSmallPer; ++k) {
    if (first + k * kSmallBlock >= last) break;
    ulonglong2* e = J.zid + cell[k];
    if (e->x == z[k]) atomicMax(&e->y, (unsigned long long)nid[k]);
  }
  flags = __reduce_or_sync(0xffffffffu, flags);
  cluster_barrier();  // all folded; the first block's words are set up
  if ((t & 31) == 0 && flags) {
    uint32_t* occ = in_block(J.occ, 0);
    if (flags & kPointNonFinite) atomicOr(in_block(&words[0], 0), kStatusNonFinite);
    if (flags & kPointOtherX) occ[1] = 1;
    if (flags & kPointOtherY) occ[3] = 1;
  }
  const uint32_t slice = (nsub + kSmallCluster - 1) / kSmallCluster, end = min(nsub, (rank + 1) * slice);
  for (uint32_t c = rank * slice + t; c < end; c += kSmallBlock) {
    Best m;
#pragma unroll
    for (int k = 0; k < kSmallCluster; ++k) {
      const ulonglong2 e = *in_block(J.zid + c, k);
      m.count += *in_block(J.count + grid_count_slot(J, c), k);
      m.take(e.x, (uint32_t)e.y);
    }
    *in_block(J.zid + c, 0) = make_ulonglong2(m.w, m.nid);
    *in_block(J.count + grid_count_slot(J, c), 0) = m.count;
  }
  cluster_barrier();
  if (rank) return;
  stamp(J, 1);
  for (int64_t i = t; i < (int64_t)J.y.nclass * J.x.n; i += kSmallBlock) rows_of(J, i);
  __syncthreads();
  for (int64_t i = t; i < (int64_t)J.y.n * J.x.n; i += kSmallBlock) window_of(J, i);
  __syncthreads();
  stamp(J, 2);
  write_seeds<false, kSmallBlock>(J, GridTiles{}, 0, 0, 1, nullptr, xy, xy_stride, llp, out.nllp);
  __syncthreads();
  stamp(J, 3);
  for (int32_t c = t >> 5; c < ncell; c += kSmallBlock / 32) cell_of(J, c);
  __syncthreads();
  write_output<kSmallBlock>(J, ncell, llp, out, 0, 1);
  if (t == 0) {  // the context's words, as the chain leaves them
    *R.status = words[0];
    *R.nllp = words[1];
    *R.ns3 = words[2];
  }
}

__global__ void k_grid_flags(const uint32_t* __restrict__ v, int64_t n, uint32_t* __restrict__ flags) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    flags[i] = v[i] != kNone ? 1u : 0u;
}
__global__ void k_grid_output_scanned(const __grid_constant__ GridJob J, const uint32_t* __restrict__ pos, int64_t ncell,
                                      const uint32_t* __restrict__ llp, GridResult R) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = t; i < ncell; i += nt)
    if (J.cellmin[i] != kNone) R.seeds[pos[i]] = J.cellmin[i];
  const uint32_t n = *R.nllp, base = *R.ns3;
  for (int64_t i = t; i < n; i += nt) R.seeds[base + i] = llp[i];
  if (t == 0) write_words(J, R, n, base);
}

// ---- batches: overlap 0 in some tile, and the output ------------------------------
// Stage 2 by sorting (tile, id) keys: the tiles' windows, then the first of
// every run of two or more (overlap > 0) or every valid one.
__global__ void k_gridb_keys(const uint32_t* __restrict__ win, GridTiles T, int64_t n, int id_bits, uint32_t none,
                             uint32_t* __restrict__ keys) {
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n; w += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t v = win[w];
    keys[w] = ((uint32_t)tile_of(T.off, T.n, w) << id_bits) | (v == kNone ? none : v);
  }
}
__global__ void k_gridb_flags(const uint32_t* __restrict__ keys, int64_t n, int id_bits, uint32_t none, GridTiles T,
                              uint32_t* __restrict__ flags, uint32_t* __restrict__ tile_count) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t k = keys[i], t = k >> id_bits;
    bool f = (k & none) != none;
    if (T.jobs[t].need_dup) f = f && (i == 0 || keys[i - 1] != k) && (i + 1 < n && keys[i + 1] == k);
    flags[i] = f ? 1u : 0u;
    if (f) atomicAdd(tile_count + t, 1u);
  }
}
__global__ void k_gridb_ids(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ flags,
                            const uint32_t* __restrict__ pos, int64_t n, int id_bits, GridTiles T, uint32_t* __restrict__ llp) {
  const uint32_t mask = (1u << id_bits) - 1u;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    if (!flags[i]) continue;
    const uint32_t id = keys[i] & mask;
    const GridJob& J = T.jobs[keys[i] >> id_bits];
    llp[pos[i]] = id;
    if (J.x.nc) mark_cells(J, J.rec, 3, id);
  }
}

// Block t: the number of tile t's cells with a result.
__global__ void __launch_bounds__(kSeedBlock) k_gridb_count(GridTiles T, uint32_t* __restrict__ s3cnt) {
  const GridJob& J = T.jobs[blockIdx.x];
  const int64_t n = (int64_t)J.x.nc * J.y.nc;
  uint32_t c = 0;
  for (int64_t i = threadIdx.x; i < n; i += kSeedBlock) c += J.cellmin[i] != kNone ? 1u : 0u;
  block_exclusive(c, &c);
  if (threadIdx.x == 0) s3cnt[blockIdx.x] = c;
}

// Block t: tile t's stage-3 ids in cell order, then its LLPs, after those of
// the tiles before it.
__global__ void __launch_bounds__(kSeedBlock) k_gridb_output(GridTiles T, const uint32_t* __restrict__ s3cnt,
                                                             const uint32_t* __restrict__ llp, const uint32_t* __restrict__ llp_off,
                                                             int64_t* __restrict__ out, int64_t* __restrict__ out_off) {
  const int t = blockIdx.x;
  const GridJob& J = T.jobs[t];
  uint32_t c = 0, s3_before;
  for (int q = threadIdx.x; q < t; q += kSeedBlock) c += __ldg(s3cnt + q);
  block_exclusive(c, &s3_before);
  const uint32_t l0 = llp_off[t], l1 = llp_off[t + 1], mine = s3cnt[t];
  int64_t at = (int64_t)s3_before + l0;
  if (threadIdx.x == 0) {
    out_off[t] = at;
    if (t == T.n - 1) out_off[T.n] = at + mine + (l1 - l0);
  }
  for (uint32_t k = threadIdx.x; k < l1 - l0; k += kSeedBlock) out[at + mine + k] = llp[l0 + k];
  const int64_t n = (int64_t)J.x.nc * J.y.nc;
  for (int64_t i = 0; i < n && mine; i += kSeedBlock) {
    const uint32_t v = i + threadIdx.x < n ? J.cellmin[i + threadIdx.x] : kNone;
    uint32_t got;
    const uint32_t p = block_exclusive(v != kNone ? 1u : 0u, &got);
    if (v != kNone) out[at + p] = v;
    at += got;
  }
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

// Whether windows (and cells whose edges count too) tile an axis in whole
// steps, so that every right edge nominally coincides with a left one.
static bool steps_tile(int32_t whalf, double step, int32_t bsize, bool cells) {
  const double steps = 2.0 * whalf / step;
  return std::fabs(steps - std::round(steps)) < 1e-6 && (!cells || bsize % 2 == 0);
}

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
  a->fmw = (1u << a->fbw) - 1u;
  a->fmc = (1u << a->fbc) - 1u;
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
  // Where every right edge nominally coincides with a left one, the classes off
  // the edges are all of one parity, read off the middle of the axis.  Only a
  // hint: a point of the other parity says so in J.occ.
  if (steps_tile(whalf, step, bsize, merged && nc > 0)) {
    int32_t cnt[4];
    const double mid = lo + 0.4637 * span;
    grid_counts_exact(*a, (uint64_t)bits_of(mid), dkey(mid), FormulaEdges{a}, cnt);
    a->par = grid_sum(*a, cnt) & 1;
    a->parmask = 1;
    const int32_t even = (a->nclass + 1) / 2;
    a->width[0] = a->par ? a->nclass - even : even;
    a->width[1] = a->nclass - a->width[0];
  } else {
    a->width[0] = a->nclass;
  }
  if (a->quick && a->linear && (merged || nc == 0)) {
    a->lcap = n + a->kl;
    a->ksum = a->kl + a->kr + a->ka + a->kb;
    int32_t at_lo[4], at_hi[4];  // no clamps but the left windows' upper one
    const int how0 = grid_counts_raw(*a, (uint64_t)bits_of(lo), at_lo), how1 = grid_counts_raw(*a, (uint64_t)bits_of(hi), at_hi);
    a->fast = how0 != 2 && how1 != 2 && at_hi[1] <= n && at_hi[2] <= nc && at_hi[3] <= nc;
    for (int f = 0; f < 4; ++f) a->fast = a->fast && at_lo[f] >= -how0;
  }
}

int grid_sizes(const owm_params& p, int64_t n, GridSizes* z) {
  const int64_t nc = p.ncols, nr = p.nrows;
  const int64_t tx = 2 * nc + 1, ty = 2 * nr + 1;
  if (tx * ty >= 0xFFFFFFFFll) return OWM_ERANGE;
  const bool cells = p.bsize > 0 && p.ngrid > 0;
  const int64_t ncg = cells ? p.ncols_grid : 0, nrg = cells ? p.nrows_grid : 0;
  // The cells' edges go with the windows' while they do not multiply the
  // sub-cells: a point then costs nothing for stage 3.  Beyond that the cells
  // get a table of their own, which no point count or window size can blow up.
  z->merged = cells && (tx + 2 * ncg) * (ty + 2 * nrg) <= std::min<int64_t>(std::max<int64_t>(4 * tx * ty, 1 << 20), 1 << 28);
  const int64_t sx = tx + (z->merged ? 2 * ncg : 0), sy = ty + (z->merged ? 2 * nrg : 0);
  z->nsub = sx * sy;
  // the sub-cells that points in no order spread over: all, or one quadrant
  const bool tile = steps_tile((uint16_t)p.wsize / 2, p.displace, (uint16_t)p.bsize, z->merged);
  z->main = tile ? ((sx + 1) / 2) * ((sy + 1) / 2) : z->nsub;
  z->counts = z->nsub + (z->main <= kGridSpreadMax ? 3 * z->main : 0);
  z->nwin = nc * nr;
  z->ncell = ncg * nrg;
  z->rows = sy * nc;
  z->edges = 24 * (nc + ncg + nr + nrg) + 16;  // keys and s-ranges, and the occupancy words
  z->chunks = ((n + 1 + 31) / 32 + kSeedChunk - 1) / kSeedChunk;
  return OWM_OK;
}

void grid_job(const owm_params& p, int64_t n, const GridSizes& z, GridJob* j) {
  GridJob& J = *j;
  std::memset(&J, 0, sizeof(J));
  const int32_t ncg = z.ncell ? (int32_t)p.ncols_grid : 0, nrg = z.ncell ? (int32_t)p.nrows_grid : 0;
  const int32_t whalf = (uint16_t)p.wsize / 2, bsize = (uint16_t)p.bsize;
  grid_axis_setup(p.bbox.min_x, p.bbox.max_x, p.displace, whalf, (int32_t)p.ncols, bsize, ncg, z.merged, &J.x);
  grid_axis_setup(p.bbox.min_y, p.bbox.max_y, p.displace, whalf, (int32_t)p.nrows, bsize, nrg, z.merged, &J.y);
  J.thr = p.min_num_points;
  J.n = (int32_t)n;
  J.need_dup = p.overlap > 0.0;
  J.sparse = n < kFoldDense * z.main;
  J.base[1] = (uint32_t)J.x.width[0] * (uint32_t)J.y.width[0];
  J.base[2] = J.base[1] + (uint32_t)J.x.width[1] * (uint32_t)J.y.width[0];
  J.base[3] = J.base[2] + (uint32_t)J.x.width[0] * (uint32_t)J.y.width[1];
  if (z.counts > z.nsub) J.spread = J.x.parmask ? J.base[1] : (uint32_t)z.nsub;
  J.fast = J.x.fast && J.y.fast && (z.merged || z.ncell == 0) ? (J.x.paired && J.y.paired ? 2 : 1) : 0;
}

namespace {
// Hands out 256-byte aligned pieces of a region, or their sizes alone.
struct Carver {
  char* base;
  size_t at = 0;
  template <class T>
  T* take(int64_t count) {
    char* q = base ? base + at : nullptr;
    at += up256((size_t)count * sizeof(T));
    return reinterpret_cast<T*>(q);
  }
};
// The edge arrays, occupancy words and ranges of a job, from a piece of
// GridSizes::edges bytes.
void carve_edges(GridJob& J, char* b) {
  auto take = [&](size_t bytes) {
    char* q = b;
    b += bytes;
    return q;
  };
  for (GridAxis* a : {&J.x, &J.y})
    for (int f = 0; f < 4; ++f) a->edge[f] = (int64_t*)take((size_t)(f < 2 ? a->n : a->nc) * 8);
  J.occ = (uint32_t*)take(16);
  for (GridAxis* a : {&J.x, &J.y}) {
    a->lo = (int32_t*)take((size_t)a->n * 4);
    a->hi = (int32_t*)take((size_t)a->n * 4);
    a->clo = (int32_t*)take((size_t)a->nc * 4);
    a->chi = (int32_t*)take((size_t)a->nc * 4);
  }
}
// What k_grid_small's tables take: the plan's pieces before the seeds.
constexpr size_t kSmallBytes = 224 * 1024;  // of a block's 227 K
size_t small_bytes(const GridPlan& g) { return (size_t)(reinterpret_cast<const char*>(g.seeds) - g.base); }
// Threads' items of k_grid_prepare: windows and cells per axis, occupancy words.
int64_t prepare_items(const owm_params& p, const GridSizes& z) {
  return (int64_t)p.ncols + p.nrows + (z.ncell ? (int64_t)p.ncols_grid + p.nrows_grid : 0) + 4;
}
}  // namespace

int grid_plan(const owm_params& p_in, int64_t n, void* scratch, GridPlan* g, bool stage1_only) {
  *g = GridPlan{};
  GridJob& J = g->job;
  owm_params p = p_in;
  if (stage1_only) p.bsize = 0;  // no cells
  if (p.ncells <= 0) return OWM_EINVAL;
  const int rc = grid_sizes(p, n, &g->z);
  if (rc) return rc;
  const GridSizes& z = g->z;
  if (scratch) grid_job(p, n, z, &J);
  g->n = n;
  g->bitmap2 = p.overlap > 0.0 && !stage1_only;
  Carver c{static_cast<char*>(scratch)};
  // cleared
  J.zid = c.take<ulonglong2>(z.nsub);
  J.count = c.take<uint32_t>(z.counts);
  if (!z.merged && z.ncell) J.cell_zid = c.take<ulonglong2>(z.ncell);
  if (g->bitmap2) {
    J.once = c.take<uint32_t>(z.chunks * kSeedChunk);
    J.twice = c.take<uint32_t>(z.chunks * kSeedChunk);
  }
  J.mark = c.take<uint8_t>(z.ncell);
  g->clear_bytes = c.at;
  // written by the kernels
  char* edges = c.take<char>(z.edges);
  if (edges) carve_edges(J, edges);
  J.rows = c.take<GridRow>(z.rows);
  if (stage1_only) {
    J.win = c.take<uint32_t>(z.nwin);
    g->bytes = c.at;
    g->base = c.base;
    return OWM_OK;
  }
  J.cellmin = c.take<uint32_t>(z.ncell);
  g->llp = c.take<uint32_t>(z.nwin);
  g->seeds = c.take<int64_t>(z.nwin + z.ncell + 1);
  if (g->bitmap2) {
    g->part = c.take<uint32_t>(z.chunks);
  } else {
    J.win = c.take<uint32_t>(z.nwin);
    g->s2_bytes = stage2_scratch_bytes(z.nwin);
    g->s2_temp = c.take<char>((int64_t)g->s2_bytes);
  }
  if (z.ncell > kOutputCells) {
    g->flags = c.take<uint32_t>(z.ncell);
    g->pos = c.take<uint32_t>(z.ncell);
    g->scan_bytes = scan_temp_bytes(z.ncell);
    g->scan_temp = c.take<char>((int64_t)g->scan_bytes);
  }
  g->bytes = c.at;
  g->base = c.base;
  return OWM_OK;
}

int grid_batch_plan(const owm_params* p, const int64_t* n, int32_t ntiles, GridSizes* z, char* base, GridBatch* g) {
  std::memset(static_cast<void*>(g), 0, sizeof(*g));  // padding too: a batch's bytes name its graph
  g->ntiles = ntiles;
  g->bitmap2 = 1;
  g->tile_bits = g->id_bits = 1;
  int64_t points = 0, nsub = 0, counts = 0, own = 0, edges = 0, maxn = 0;
  for (int32_t k = 0; k < ntiles; ++k) {
    const int rc = grid_sizes(p[k], n[k], &z[k]);
    if (rc) return rc;
    if (!(p[k].overlap > 0.0)) g->bitmap2 = 0;
    points += n[k];
    maxn = std::max(maxn, n[k]);
    nsub += z[k].nsub;
    counts += z[k].counts;
    own += z[k].merged ? 0 : z[k].ncell;
    edges += (z[k].edges + 15) & ~(int64_t)15;
    g->items += prepare_items(p[k], z[k]);
    g->rows += z[k].rows;
    g->wins += z[k].nwin;
    g->row_blocks += (z[k].rows + 255) / 256;
    g->win_blocks += (z[k].nwin + 255) / 256;
    g->chunks += z[k].chunks;
    g->cells += z[k].ncell;
  }
  // enough fold blocks to fill the chip twice, of 256 to 4096 points
  g->chunk = (int32_t)std::min<int64_t>(kTileChunk, std::max<int64_t>(256, (points / (152 * kFoldBlocks * 2) + 255) / 256 * 256));
  for (int32_t k = 0; k < ntiles; ++k) g->folds += (n[k] + g->chunk - 1) / g->chunk;
  if (g->folds >= 0x7FFFFFFFll || g->chunks >= 0x7FFFFFFFll || g->cells >= 0x7FFFFFFFll * 8) return OWM_ERANGE;
  while (((uint64_t)1 << g->tile_bits) < (uint64_t)ntiles) ++g->tile_bits;
  while (((uint64_t)1 << g->id_bits) <= (uint64_t)maxn + 1) ++g->id_bits;
  if (g->tile_bits + g->id_bits > 32) return OWM_ERANGE;  // split the batch

  Carver c{base};
  g->zid = c.take<char>(nsub * 16);
  g->count = c.take<char>(counts * 4);
  g->cell_zid = c.take<char>(own * 16);
  g->bitmap = g->bitmap2 ? c.take<uint32_t>(2 * g->chunks * kSeedChunk) : nullptr;
  g->mark = c.take<char>(g->cells);
  g->cnt2 = c.take<uint32_t>(ntiles + 1);
  g->words = c.take<uint32_t>(64);
  g->clear_bytes = c.at;
  g->jobs = c.take<GridJob>(ntiles);
  for (auto** v : {&g->item_off, &g->fold_off, &g->row_off, &g->win_off, &g->winb_off, &g->chunk_off, &g->cell_off})
    *v = c.take<int64_t>(ntiles + 1);
  g->table_bytes = c.at - g->clear_bytes;
  g->edges = c.take<char>(edges);
  g->row_mem = c.take<char>(g->rows * (int64_t)sizeof(GridRow));
  g->cellmin = c.take<char>(g->cells * 4);
  g->llp = c.take<uint32_t>(g->wins);
  g->llp_off = c.take<uint32_t>(ntiles + 1);
  g->s3cnt = c.take<uint32_t>(ntiles + 1);
  g->out = c.take<int64_t>(g->wins + g->cells + 1);
  g->out_off = c.take<int64_t>(ntiles + 1);
  if (g->bitmap2) {
    g->part = c.take<uint32_t>(g->chunks);
  } else {
    g->win = c.take<uint32_t>(g->wins);
    g->k0 = c.take<uint32_t>(g->wins);
    g->k1 = c.take<uint32_t>(g->wins);
    g->flags = c.take<uint32_t>(g->wins);
    g->pos = c.take<uint32_t>(g->wins);
    g->sort_bytes = radix_sort_temp_bytes(g->wins);
    g->sort_temp = c.take<char>((int64_t)g->sort_bytes);
    g->scan_bytes = scan_temp_bytes(std::max<int64_t>(g->wins, ntiles + 1));
    g->scan_temp = c.take<char>((int64_t)g->scan_bytes);
  }
  g->bytes = c.at;
  g->base = base;
  return OWM_OK;
}

void grid_batch_tables(const owm_params* p, const int64_t* n, const GridSizes* z, const double* const* rec, const GridBatch& g,
                       char* host) {
  auto at = [&](const void* device) { return host + (static_cast<const char*>(device) - reinterpret_cast<const char*>(g.jobs)); };
  GridJob* jobs = reinterpret_cast<GridJob*>(host);
  int64_t *items = (int64_t*)at(g.item_off), *folds = (int64_t*)at(g.fold_off), *rows = (int64_t*)at(g.row_off),
          *wins = (int64_t*)at(g.win_off), *winb = (int64_t*)at(g.winb_off), *chunks = (int64_t*)at(g.chunk_off), *cells = (int64_t*)at(g.cell_off);
  items[0] = folds[0] = rows[0] = wins[0] = winb[0] = chunks[0] = cells[0] = 0;
  int64_t sub = 0, counts = 0, own = 0, edges = 0, row_mem = 0;
  for (int32_t k = 0; k < g.ntiles; ++k) {
    GridJob& J = jobs[k];
    grid_job(p[k], n[k], z[k], &J);
    J.rec = rec[k];
    J.zid = (ulonglong2*)g.zid + sub;
    J.count = (uint32_t*)g.count + counts;
    sub += z[k].nsub;
    counts += z[k].counts;
    if (!z[k].merged && z[k].ncell) {
      J.cell_zid = (ulonglong2*)g.cell_zid + own;
      own += z[k].ncell;
    }
    if (g.bitmap2) {
      J.once = g.bitmap + chunks[k] * kSeedChunk;
      J.twice = g.bitmap + (g.chunks + chunks[k]) * kSeedChunk;
    } else {
      J.win = g.win + wins[k];
    }
    J.mark = (uint8_t*)g.mark + cells[k];
    carve_edges(J, g.edges + edges);
    edges += (z[k].edges + 15) & ~(int64_t)15;
    J.rows = (GridRow*)g.row_mem + row_mem;
    row_mem += z[k].rows;
    J.cellmin = (uint32_t*)g.cellmin + cells[k];
    items[k + 1] = items[k] + prepare_items(p[k], z[k]);
    folds[k + 1] = folds[k] + (n[k] + g.chunk - 1) / g.chunk;
    rows[k + 1] = rows[k] + (z[k].rows + 255) / 256;
    wins[k + 1] = wins[k] + z[k].nwin;
    winb[k + 1] = winb[k] + (z[k].nwin + 255) / 256;
    chunks[k + 1] = chunks[k] + z[k].chunks;
    cells[k + 1] = cells[k] + z[k].ncell;
  }
}

int grid_batch_run(const GridBatch& g, cudaStream_t s, int64_t* launches) {
  GridJob none;
  std::memset(&none, 0, sizeof(none));
  auto tiles = [&](const int64_t* off) { return GridTiles{g.jobs, off, g.ntiles}; };
  const int64_t n16 = (int64_t)(g.clear_bytes / 16);
  OWM_LAUNCH("k_grid_prepare", s, k_grid_prepare<true><<<blocks_for(std::max(n16, g.items), 152 * 8), 256, 0, s>>>(
      none, tiles(g.item_off), g.items, (uint4*)g.base, n16, g.words));
  OWM_LAUNCH("k_grid_fold_tiles", s, k_grid_fold_tiles<<<(unsigned)((g.folds + kTileStripes - 1) / kTileStripes * kTileStripes), kFoldBlock, 0, s>>>(tiles(g.fold_off), g.chunk, g.words));
  count_launch(launches, 2);
  if (g.wins > 0) {
    OWM_LAUNCH("k_grid_rows", s, k_grid_rows<true><<<(unsigned)g.row_blocks, 256, 0, s>>>(none, tiles(g.row_off)));
    OWM_LAUNCH("k_grid_windows", s, k_grid_windows<true><<<(unsigned)g.win_blocks, 256, 0, s>>>(none, tiles(g.winb_off)));
    count_launch(launches, 2);
  }
  if (g.bitmap2) {
    OWM_LAUNCH("k_grid_seed_count", s, k_grid_seed_count<<<(unsigned)g.chunks, kSeedBlock, 0, s>>>(
        g.bitmap + g.chunks * kSeedChunk, g.part));
    OWM_LAUNCH("k_grid_seeds", s, k_grid_seeds<true><<<(unsigned)g.chunks, kSeedBlock, 0, s>>>(
        none, tiles(g.chunk_off), g.part, nullptr, 3, g.llp, g.llp_off));
    count_launch(launches, 2);
  } else {
    const uint32_t ids = (1u << g.id_bits) - 1u;
    const unsigned nb = blocks_for(g.wins, 152 * 32);
    OWM_LAUNCH("k_gridb_keys", s, k_gridb_keys<<<nb, 256, 0, s>>>(g.win, tiles(g.win_off), g.wins, g.id_bits, ids, g.k0));
    bool alt = false;
    if (g.wins > 0)
      OWM_CUDA_TRY(radix_sort(g.k0, nullptr, g.k1, nullptr, g.wins, g.tile_bits + g.id_bits, false, g.sort_temp, g.sort_bytes, s,
                            &alt, launches));
    const uint32_t* keys = alt ? g.k1 : g.k0;
    OWM_LAUNCH("k_gridb_flags", s, k_gridb_flags<<<nb, 256, 0, s>>>(keys, g.wins, g.id_bits, ids, tiles(g.win_off), g.flags, g.cnt2));
    if (g.wins > 0) OWM_CUDA_TRY(exclusive_scan_u32(g.flags, g.pos, g.wins, nullptr, g.scan_temp, g.scan_bytes, s, launches));
    OWM_LAUNCH("k_gridb_ids", s, k_gridb_ids<<<nb, 256, 0, s>>>(keys, g.flags, g.pos, g.wins, g.id_bits, tiles(g.win_off), g.llp));
    OWM_CUDA_TRY(exclusive_scan_u32(g.cnt2, g.llp_off, g.ntiles + 1, nullptr, g.scan_temp, g.scan_bytes, s, launches));
    count_launch(launches, 3);
  }
  if (g.cells > 0) {
    OWM_LAUNCH("k_grid_cells", s, k_grid_cells<true><<<(unsigned)((g.cells + 7) / 8), 256, 0, s>>>(none, tiles(g.cell_off), g.cells));
    count_launch(launches);
  }
  OWM_LAUNCH("k_gridb_count", s, k_gridb_count<<<(unsigned)g.ntiles, kSeedBlock, 0, s>>>(tiles(g.cell_off), g.s3cnt));
  OWM_LAUNCH("k_gridb_output", s, k_gridb_output<<<(unsigned)g.ntiles, kSeedBlock, 0, s>>>(tiles(g.cell_off), g.s3cnt, g.llp, g.llp_off,
                                                                                     g.out, g.out_off));
  count_launch(launches, 2);
  OWM_CUDA_TRY(cudaGetLastError());
  return OWM_OK;
}

int grid_prepare(const GridPlan& g, const owm_params& p, uint32_t* status, cudaStream_t s, int64_t* launches) {
  const int64_t n16 = (int64_t)(g.clear_bytes / 16);
  OWM_LAUNCH("k_grid_prepare", s, k_grid_prepare<false><<<blocks_for(n16, 152 * 8), 256, 0, s>>>(
      g.job, GridTiles{}, prepare_items(p, g.z), (uint4*)g.base, n16, status));
  count_launch(launches);
  OWM_CUDA_TRY(cudaGetLastError());
  return OWM_OK;
}

namespace {
// A call's time with the shared tables and without, by points per sub-cell that
// points in no order spread over: 41 (65 K points) 46 and 42 us, 55 (60 K) 45 and
// 43, 83 (200 K) 50 and 50, 115 (400 K) 45 and 57, 137 (100 K) 40 and 43, 833 (2 M)
// 55 and 122, 6200 (20 M) 209 and 904.
constexpr int64_t kFewCells = 8192;  // 192 KB of tables
bool fold_few(const GridPlan& g) {
  return g.z.nsub <= kFewCells && g.n >= 96 * g.z.main;
}
}  // namespace

int grid_fold(const GridPlan& g, const GridPoints& pts, uint32_t* status, cudaStream_t s, int64_t* launches) {
  const GridJob& J = g.job;
  if (fold_few(g)) {
    using Few = void (*)(GridJob, GridPoints, uint32_t, uint32_t*);
    const Few kernel = pts.stride == 4 ? k_grid_fold_few<4> : pts.stride == 3 ? k_grid_fold_few<3> : k_grid_fold_few<0>;
    OWM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)few_bytes(kFewCells)));
    OWM_LAUNCH("k_grid_fold", s, OWM_CUDA_TRY(chain_smem(kernel, blocks_for(J.n, 152, kFewBlock * kFewPer), kFewBlock,
                                                         few_bytes(g.z.nsub), s, J, pts, (uint32_t)g.z.nsub, status)));
    count_launch(launches);
    OWM_CUDA_TRY(cudaGetLastError());
    return OWM_OK;
  }
  const unsigned nb = blocks_for(J.n, 152 * kFoldBlocks, kFoldBlock);
  using Kernel = void (*)(GridJob, GridPoints, uint32_t*);
  static const Kernel kernels[3][3][2] = {
      {{k_grid_fold<0, 0, true>, k_grid_fold<0, 0, true>}, {k_grid_fold<0, 1, false>, k_grid_fold<0, 1, true>}, {k_grid_fold<0, 2, false>, k_grid_fold<0, 2, true>}},
      {{k_grid_fold<3, 0, true>, k_grid_fold<3, 0, true>}, {k_grid_fold<3, 1, false>, k_grid_fold<3, 1, true>}, {k_grid_fold<3, 2, false>, k_grid_fold<3, 2, true>}},
      {{k_grid_fold<4, 0, true>, k_grid_fold<4, 0, true>}, {k_grid_fold<4, 1, false>, k_grid_fold<4, 1, true>}, {k_grid_fold<4, 2, false>, k_grid_fold<4, 2, true>}}};
  const Kernel kernel = kernels[pts.stride == 4 ? 2 : pts.stride == 3 ? 1 : 0][J.fast][J.sparse];
  OWM_LAUNCH("k_grid_fold", s, OWM_CUDA_TRY(chain(kernel, nb, kFoldBlock, s, J, pts, status)));
  count_launch(launches);
  OWM_CUDA_TRY(cudaGetLastError());
  return OWM_OK;
}

// 32 K points take 39 us a call this way and 43 as a chain, 20 K 34 and 40, 1 K
// 28 and 36; 10 K more points add 4 us here and 1 there.  Cells with a table of
// their own, and stage 2 by sorting, go by the chain.
bool grid_is_small(const GridPlan& g) {
  return g.bitmap2 && g.n <= kSmallPoints && (g.z.merged || g.z.ncell == 0) && small_bytes(g) <= kSmallBytes;
}

int grid_small(const GridPlan& g, const owm_params& p, const GridPoints& pts, const double* xy, int xy_stride,
               const GridResult& out, cudaStream_t s, int64_t* launches) {
  const auto kernel = pts.stride == 4 ? k_grid_small<4> : k_grid_small<3>;
  OWM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallBytes));
  OWM_LAUNCH("k_grid_small", s, kernel<<<kSmallCluster, kSmallBlock, small_bytes(g), s>>>(
      g.job, pts, g.base, prepare_items(p, g.z), (int64_t)(g.clear_bytes / 16), (uint32_t)g.z.nsub, xy, xy_stride,
      (int32_t)g.z.ncell, reinterpret_cast<const char*>(g.llp) - g.base, out));
  count_launch(launches);
  OWM_CUDA_TRY(cudaGetLastError());
  return OWM_OK;
}

int grid_windows(const GridPlan& g, cudaStream_t s, int64_t* launches) {
  const GridJob& J = g.job;
  OWM_LAUNCH("k_grid_rows", s, OWM_CUDA_TRY(chain(k_grid_rows<false>, (unsigned)((g.z.rows + 255) / 256), 256, s, J, GridTiles{})));
  OWM_LAUNCH("k_grid_windows", s, OWM_CUDA_TRY(chain(k_grid_windows<false>, (unsigned)((g.z.nwin + 255) / 256), 256, s, J, GridTiles{})));
  count_launch(launches, 2);
  OWM_CUDA_TRY(cudaGetLastError());
  return OWM_OK;
}

int grid_stage2(const GridPlan& g, const owm_params& p, const double* xy, int xy_stride, uint32_t* d_nllp,
                cudaStream_t s, int64_t* launches) {
  const GridJob& J = g.job;
  if (g.bitmap2) {
    // up to 32 chunks (1 M ids) each block counts the words before its own: one
    // launch less
    const unsigned chunks = (unsigned)g.z.chunks;
    const bool count = chunks > 32;
    if (count)
      OWM_LAUNCH("k_grid_seed_count", s, OWM_CUDA_TRY(chain(k_grid_seed_count, chunks, kSeedBlock, s, J.twice, g.part)));
    OWM_LAUNCH("k_grid_seeds", s, OWM_CUDA_TRY(chain(k_grid_seeds<false>, chunks, kSeedBlock, s, J, GridTiles{},
                                                     count ? g.part : nullptr, xy, xy_stride, g.llp, d_nllp)));
    count_launch(launches, 1 + count);
  } else {
    // overlap 0 keeps every valid minimum, repeated sentinel ids included: by sorting
    const int rc = run_stage2(J.win, g.z.nwin, g.n, p.overlap, g.llp, d_nllp, g.s2_temp, g.s2_bytes, s, launches);
    if (rc) return rc;
    if (g.z.ncell) {
      OWM_LAUNCH("k_grid_mark", s, k_grid_mark<<<blocks_for(g.z.nwin, 152 * 8), 256, 0, s>>>(J, xy, xy_stride, g.llp, d_nllp));
      count_launch(launches);
    }
  }
  OWM_CUDA_TRY(cudaGetLastError());
  return OWM_OK;
}

int grid_stage3(const GridPlan& g, const GridResult& out, cudaStream_t s, int64_t* launches) {
  const GridJob& J = g.job;
  if (g.z.ncell > 0) {
    OWM_LAUNCH("k_grid_cells", s, OWM_CUDA_TRY(chain(k_grid_cells<false>, (unsigned)((g.z.ncell + 7) / 8), 256, s, J, GridTiles{},
                                                     g.z.ncell)));
    count_launch(launches);
  }
  if (g.z.ncell <= kOutputCells) {
    OWM_LAUNCH("k_grid_output", s, OWM_CUDA_TRY(chain(k_grid_output, blocks_for(g.z.nwin / 4 + g.z.ncell, 64), kSeedBlock, s, J,
                                                      g.z.ncell, g.llp, out)));
    count_launch(launches);
  } else {
    OWM_LAUNCH("k_grid_flags", s, k_grid_flags<<<blocks_for(g.z.ncell, 152 * 8), 256, 0, s>>>(J.cellmin, g.z.ncell, g.flags));
    count_launch(launches);
    OWM_CUDA_TRY(exclusive_scan_u32(g.flags, g.pos, g.z.ncell, out.ns3, g.scan_temp, g.scan_bytes, s, launches));
    OWM_LAUNCH("k_grid_output", s, k_grid_output_scanned<<<blocks_for(g.z.nwin + g.z.ncell, 152 * 8), 256, 0, s>>>(
        J, g.pos, g.z.ncell, g.llp, out));
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
    if (!a.fast) continue;
    uint32_t h;
    int32_t t[4];
    const int32_t cls = a.paired ? grid_class_fast<true>(a, b, &h, t) : grid_class_fast<false>(a, b, &h, t);
    if (h & kGridOutside) {
      if (how != 2) return 1;
    } else if (grid_settle_fast(a, dkey(p[i]), h, t, FormulaEdges{&a}, cls) != grid_sum(a, counts + 4 * i)) {
      return 1;
    }
  }
  return 0;
}

// Window grid: the whole path of one cloud without a spatial hierarchy.
//
// Along one axis the stage-1 windows (L_j, R_j) and the stage-3 cells
// (A_i, B_i) are open intervals whose edges do not decrease with their index.
// For a coordinate p let
//     s(p) = #{L_j < p} + #{R_j <= p} + #{A_i < p} + #{B_i <= p}.
// s does not decrease with p, and an interval (l, r) of either family contains
// p exactly when s(l+) <= s(p) <= s(r-), with l+ / r- the next double above l /
// below r.  So every point falls in one (s_x, s_y) sub-cell, and every window
// and every cell is a rectangle of sub-cells.  The path is then: one pass over
// the points that keeps each sub-cell's count and (z, id)-minimum (the
// reference's O3 memo, optim3_func.cpp:255-307, on the sub-cells instead of
// quadtree nodes), and rectangle reductions for stage 1 and stage 3.
#pragma once

#include "owm_query.cuh"

namespace owm {

enum GridFamily { kFamL = 0, kFamR = 1, kFamA = 2, kFamB = 3 };

// One axis.  A coordinate's sub-cell is found by arithmetic, not by a table or
// a search: its position v (32 bits, a fixed-point offset from the axis's
// origin) times a constant is its place in window (cell) steps, whose integer
// part is the number of edges passed.  A place within kGridGuard units of an
// edge's nominal one is settled by comparing with the edge itself.
struct __align__(16) GridAxis {
  // The fast form's constants (grid_class_fast), for coordinates in [lo, hi] off
  // the edges: place = mulhi(position above lo, m) + q by family, t = place >> fb,
  // s = min(tl, lcap) + tr + ta + tb - ksum.  80 bytes that a batch's fold reads
  // in five 16-byte words.
  int64_t lo0;               // lo's bits (linear) or whole quanta (general)
  uint64_t span;             // hi's minus lo's
  int32_t sh;                // linear: bits shifted out; general: biased exponent of the quantum + 52
  uint32_t mw, mc;           // steps per position, times 2^(32 + fb): windows, cells
  uint32_t qw;               // place of lo: L
  uint32_t qc;               // place of lo: A
  int32_t fbw, fbc;          // fraction bits of a place
  int32_t lcap;
  int32_t ksum, par;         // par: the main parity of s
  uint32_t fmw, fmc;         // masks of a place's fraction
  uint32_t qr, qb;           // places of lo: R, B
  int32_t parmask, pad;      // 1: points off the edges all have s & 1 == par
  // the rest of the form for [lo, hi]
  int32_t kl, kr, ka, kb;    // edge counts at place 0
  int32_t paired;            // R and B places lie where L and A places do: one place for both
  int32_t fast;              // the fast form holds over all of [lo, hi]
  int64_t f0;                // position 0: a double's bits (linear) or whole quanta (general)
  uint32_t c[4];             // place of position 0 by family, bias and guard added
  int32_t kw, kc;            // bias: count = (place >> fb) - bias, clamped to [0, n]
  int32_t n, nc;             // windows, cells
  int32_t quick;             // 0: no fixed-point form (every coordinate is searched)
  int32_t linear;            // 1: the range lies in one positive binade, a double's bits are linear in it
  int32_t merged;            // s counts the cells' edges too
  int32_t nclass;            // values of s
  int32_t width[2];          // stored classes: of the main parity, of the other; all, none (parmask 0)
  double wbase, step, wr;    // L_j = (wbase + j * step) - wr, R_j = ... + wr
  double cbase, cr;          // A_i = (cbase + i * bsize) - cr, B_i = ... + cr
  int32_t bsize;
  const int64_t* edge[4];    // order keys of the edges, by family (device)
  int32_t *lo, *hi, *clo, *chi;  // s-range of every window and cell (device; merged cells only)
};

// Places are compared with nominal ones in units of 2^-fb steps; one position
// is at most one unit.  An edge's double lies within 2.5 units of the exact
// arithmetic progression (its roundings after the first edge's: j * step, the
// sum, the half width, each at most half an ulp, an ulp at most one position),
// flooring the position and the product adds 2, rounding the constants and
// the origin 2.  Places further than the guard from an edge's nominal place
// are therefore on the same side of the edge as the coordinate is.
constexpr uint32_t kGridGuard = 16;
// Fewest fraction bits of the fixed-point form: a step of 256 units, an eighth of
// which lies within the guard of an edge.
constexpr int32_t kGridMinFrac = 8;
static_assert((1u << kGridMinFrac) >= 4 * kGridGuard, "the guards of neighbouring edges do not meet");

__host__ __device__ __forceinline__ double grid_add(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dadd_rn(a, b);
#else
  return a + b;
#endif
}
__host__ __device__ __forceinline__ double grid_mul(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}

// Edge j of a family, as an order key; the reference's arithmetic (stage 1:
// optim3_func.cpp:318-324, 544-555; stage 3: :310-316, 630-651), each
// operation rounded by itself.
__host__ __device__ __forceinline__ int64_t grid_edge(const GridAxis& a, int fam, int32_t j) {
  if (fam < 2) {
    const double c = grid_add(a.wbase, grid_mul((double)j, a.step));
    return dkey(grid_add(c, fam == kFamL ? -a.wr : a.wr));
  }
  const double c = grid_add(a.cbase, (double)(j * a.bsize));
  return dkey(grid_add(c, fam == kFamA ? -a.cr : a.cr));
}

// Whether an edge lies below a coordinate: strictly for the left edges, not
// above it for the right ones.
__host__ __device__ __forceinline__ bool grid_passed(int fam, int64_t edge, int64_t key) {
  return (fam & 1) ? edge <= key : edge < key;
}

// Position of the double with these bits; false outside the axis's range
// (also for NaN and infinities).
__host__ __device__ __forceinline__ bool grid_position(const GridAxis& a, uint64_t bits, uint32_t* v) {
  uint64_t d;
  bool ok = a.quick != 0;
  if (a.linear) {
    d = (bits - (uint64_t)a.f0) >> a.sh;
  } else {
    const int32_t e = (int32_t)((bits >> 52) & 0x7FF);
    const uint64_t m = (bits & 0xFFFFFFFFFFFFFull) | (e ? 0x10000000000000ull : 0ull);
    const int32_t s = a.sh - (e ? e : 1);
    ok = ok && s >= 0 && e != 0x7FF;
    const int64_t f = s > 63 || s < 0 ? 0 : (int64_t)(m >> s);
    d = (uint64_t)(((int64_t)bits < 0 ? -f : f) - a.f0);
  }
  *v = (uint32_t)d;
  return ok && (d >> 32) == 0;
}

__host__ __device__ __forceinline__ uint32_t grid_mulhi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

__host__ __device__ __forceinline__ int32_t grid_clamp(int32_t v, int32_t n) { return v < 0 ? 0 : (v > n ? n : v); }

// Edges of one family passed at position v, and whether the place is near one.
__host__ __device__ __forceinline__ int32_t grid_count(const GridAxis& a, int fam, uint32_t v, bool* near) {
  const bool win = fam < 2;
  const int32_t fb = win ? a.fbw : a.fbc;
  const uint32_t h = grid_mulhi(v, win ? a.mw : a.mc) + a.c[fam];
  *near = (h & ((1u << fb) - 1u)) < 2 * kGridGuard;
  return (int32_t)(h >> fb) - (win ? a.kw : a.kc);
}

// Edge count of family f at an order key, exactly.  v: the key's position, where
// it has one (ok).  edge_of(fam, j) gives the edges' order keys.
template <class EdgeOf>
__host__ __device__ __forceinline__ int32_t grid_count_exact(const GridAxis& a, int f, bool ok, uint32_t v, int64_t key,
                                                             EdgeOf edge_of) {
  const int32_t n = f < 2 ? a.n : a.nc;
  if (ok) {
    bool near;
    int32_t k = grid_count(a, f, v, &near);
    if (near && k >= 1 && k <= n) k -= grid_passed(f, edge_of(f, k - 1), key) ? 0 : 1;
    return grid_clamp(k, n);
  }
  int32_t lo = 0, hi = n;
  while (lo < hi) {
    const int32_t mid = (lo + hi) >> 1;
    if (grid_passed(f, edge_of(f, mid), key)) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// All four of a coordinate.
template <class EdgeOf>
__host__ __device__ __forceinline__ void grid_counts_exact(const GridAxis& a, uint64_t bits, int64_t key, EdgeOf edge_of,
                                                           int32_t cnt[4]) {
  uint32_t v;
  const bool ok = grid_position(a, bits, &v);
  for (int f = 0; f < 4; ++f) cnt[f] = grid_count_exact(a, f, ok, v, key, edge_of);
}

// The four edge counts of a coordinate in [lo, hi], not yet clamped to their
// upper ends.  0: exact.  1: near an edge, each at most one too high
// (grid_settle).  2: not in [lo, hi], cnt means nothing.
// Off the edges no count is negative in [lo, hi]: the first edges lie at most
// one step above lo.  Where windows and cells tile the axis in whole steps one
// place serves left and right edges.
__host__ __device__ __forceinline__ int grid_counts_raw(const GridAxis& a, uint64_t bits, int32_t cnt[4]) {
  uint32_t v;
  bool in;
  if (a.linear) {
    const uint64_t d = bits - (uint64_t)a.lo0;
    in = d <= a.span;
    v = (uint32_t)(d >> a.sh);
  } else {
    in = grid_position(a, bits, &v);
    v -= 1u << 30;
    in = in && v <= (uint32_t)a.span;
  }
  const uint32_t hl = grid_mulhi(v, a.mw) + a.qw, ha = grid_mulhi(v, a.mc) + a.qc;
  bool off = (hl & a.fmw) >= 2 * kGridGuard && (ha & a.fmc) >= 2 * kGridGuard;
  uint32_t hr = hl, hb = ha;
  if (!a.paired) {
    hr = grid_mulhi(v, a.mw) + a.qr;
    hb = grid_mulhi(v, a.mc) + a.qb;
    off = off && (hr & a.fmw) >= 2 * kGridGuard && (hb & a.fmc) >= 2 * kGridGuard;
  }
  cnt[0] = (int32_t)(hl >> a.fbw) - a.kl;
  cnt[1] = (int32_t)(hr >> a.fbw) - a.kr;
  cnt[2] = (int32_t)(ha >> a.fbc) - a.ka;
  cnt[3] = (int32_t)(hb >> a.fbc) - a.kb;
  return !in ? 2 : off ? 0 : 1;
}

// Counts of a coordinate by all of the above.
template <class EdgeOf>
__host__ __device__ __forceinline__ int grid_counts(const GridAxis& a, uint64_t bits, EdgeOf edge_of, int32_t cnt[4]) {
  const int how = grid_counts_raw(a, bits, cnt);
  if (how == 2) return how;
#pragma unroll
  for (int f = 0; f < 4; ++f) cnt[f] = cnt[f] < (f < 2 ? a.n : a.nc) + how ? cnt[f] : (f < 2 ? a.n : a.nc) + how;
  if (how == 0) return how;
  double d;
#ifdef __CUDA_ARCH__
  d = __longlong_as_double((long long)bits);
#else
  __builtin_memcpy(&d, &bits, 8);
#endif
  const int64_t key = dkey(d);
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    const int32_t n = f < 2 ? a.n : a.nc, k = cnt[f];
    if (n > 0)
      cnt[f] = grid_clamp(k, n) - (k >= 1 && k <= n && !grid_passed(f, edge_of(f, grid_clamp(k - 1, n - 1)), key));
    else
      cnt[f] = 0;
  }
  return how;
}

__host__ __device__ __forceinline__ int32_t grid_sum(const GridAxis& a, const int32_t cnt[4]) {
  return cnt[0] + cnt[1] + (a.merged ? cnt[2] + cnt[3] : 0);
}

// Class of a coordinate on an axis with the fast form, where *how is 0.  Near a
// window edge (kGridNearWindow), a cell edge (kGridNearCell) or both, the edges
// that its places t (by family) end at still have to be looked at
// (grid_settle_fast); kGridOutside: not in [lo, hi].  kPaired: the axis is
// (R shares L's place, B shares A's).  a: a GridAxis or a copy of its first 80
// bytes.
constexpr uint32_t kGridNearWindow = 1, kGridNearCell = 2, kGridOutside = 4;
template <bool kPaired, class Axis>
__host__ __device__ __forceinline__ int32_t grid_class_fast(const Axis& a, uint64_t bits, uint32_t* how, int32_t t[4]) {
  const uint64_t d = bits - (uint64_t)a.lo0;
  const uint32_t v = (uint32_t)(d >> a.sh);
  const uint32_t mw = grid_mulhi(v, a.mw), mc = grid_mulhi(v, a.mc);
  const uint32_t hl = mw + a.qw, ha = mc + a.qc;
  bool nw = (hl & a.fmw) < 2 * kGridGuard, nc = (ha & a.fmc) < 2 * kGridGuard;
  t[0] = t[1] = (int32_t)(hl >> a.fbw);
  t[2] = t[3] = (int32_t)(ha >> a.fbc);
  if (!kPaired) {
    const uint32_t hr = mw + a.qr, hb = mc + a.qb;
    nw |= (hr & a.fmw) < 2 * kGridGuard;
    nc |= (hb & a.fmc) < 2 * kGridGuard;
    t[1] = (int32_t)(hr >> a.fbw);
    t[3] = (int32_t)(hb >> a.fbc);
  }
  *how = (d > a.span ? kGridOutside : 0u) | (nw ? kGridNearWindow : 0u) | (nc ? kGridNearCell : 0u);
  return (t[0] < a.lcap ? t[0] : a.lcap) + t[1] + t[2] + t[3] - a.ksum;
}

// The class s that the fast form gave near an edge counts the edges at its
// places as passed: takes back those that are not.  (Linear axes: a
// coordinate's bits are its order key.)
template <class EdgeOf>
__host__ __device__ __forceinline__ int32_t grid_settle_fast(const GridAxis& a, int64_t key, uint32_t how, const int32_t t[4],
                                                             EdgeOf edge_of, int32_t s) {
  if (how & kGridNearWindow) {
    const int32_t l = t[0] - a.kl - 1, r = t[1] - a.kr - 1;
    const bool has_l = l >= 0 && l < a.n, has_r = r >= 0 && r < a.n;
    const int64_t el = has_l ? edge_of(kFamL, l) : 0, er = has_r ? edge_of(kFamR, r) : 0;
    s -= (has_l && !(el < key)) + (has_r && !(er <= key));
  }
  if (how & kGridNearCell) {
    const int32_t l = t[2] - a.ka - 1, r = t[3] - a.kb - 1;
    const bool has_l = l >= 0 && l < a.nc, has_r = r >= 0 && r < a.nc;
    const int64_t el = has_l ? edge_of(kFamA, l) : 0, er = has_r ? edge_of(kFamB, r) : 0;
    s -= (has_l && !(el < key)) + (has_r && !(er <= key));
  }
  return s;
}
struct GridFastAxis {
  int64_t lo0;
  uint64_t span;
  int32_t sh;
  uint32_t mw, mc, qw, qc;
  int32_t fbw, fbc, lcap, ksum, par;
  uint32_t fmw, fmc, qr, qb;
  int32_t parmask, pad;
};
static_assert(sizeof(GridFastAxis) == 80, "the first five 16-byte words of a GridAxis");

// Count and (z, id)-minimum of a box, all zero when empty: w is the inverted,
// sign-flipped order key of z and nid the inverted id, so the lexicographic
// maximum of (w, nid) is the (z, id)-minimum.
struct __align__(16) GridRow {
  unsigned long long w;
  uint32_t nid, count;
};

// Where windows and cells tile the axes in whole steps (overlap 0.8: W = 5
// steps), every right edge nearly coincides with a left one and every second
// class is a few ulps wide and all but empty.  Sub-cells of such an axis
// (parmask) are stored by parity, the main one first, s >> 1 within it: the
// full sub-cells of two such axes lie side by side, a quarter of the table.
struct __align__(16) GridJob {
  GridAxis x, y;
  uint32_t base[4];      // first sub-cell of quadrant 2 * (y not main) + (x not main)
  int32_t fast;          // both axes have the fast form: 2 paired, 1 not
  uint32_t spread;       // the first sub-cells, whose counts lie 16 bytes apart
  ulonglong2* zid;       // [sub-cells] (w, nid)
  uint32_t* count;       // [sub-cells], at grid_count_slot
  ulonglong2* cell_zid;  // [cells] (w, nid), when the cells are not merged
  GridRow* rows;         // [y.nclass][x.n], main parity first
  uint32_t* occ;         // [4] words: x main / other, y main / other classes hold points
  uint8_t* mark;         // [cells] an LLP lies in the cell
  uint32_t* cellmin;     // [cells] stage-3 id or kNone
  uint32_t* once;        // stage-2 bitmaps over ids 0..n
  uint32_t* twice;
  uint32_t* win;         // [windows] stage-1 ids (kept when overlap is 0)
  uint32_t thr;
  int32_t n;
  const double* rec;     // batches: the tile's points (plain x, y, z)
  int16_t need_dup;      // overlap > 0: LLPs are ids of two or more windows
  int16_t sparse;        // fewer than kFoldDense points a full sub-cell
  unsigned long long* stamps;  // [kGridStamps] nanoseconds at the phases' ends, or null
};
// Phase stamps: start, index done, stage 1, stage 2, stage 3 and output done.
constexpr int kGridStamps = 5;

// Points as the fold reads them: records of `stride` doubles (4: 32-byte records
// x, y, z, pad; 3: plain x, y, z), point i with id i + 1; or (stride 0) a tree's
// sorted order keys and ids.
struct GridPoints {
  const double* rec = nullptr;
  int stride = 0;
  const int64_t *xk = nullptr, *yk = nullptr, *zk = nullptr;
  const uint32_t* id = nullptr;
};

// The tiles of a batch as a kernel sees them: off[t] is tile t's first item.
struct GridTiles {
  const GridJob* jobs = nullptr;
  const int64_t* off = nullptr;
  int32_t n = 0;
};

// Stored index of sub-cell (sx, sy).
__host__ __device__ __forceinline__ uint32_t grid_cell(const GridJob& J, int32_t sx, int32_t sy) {
  const int qx = (sx ^ J.x.par) & J.x.parmask, qy = (sy ^ J.y.par) & J.y.parmask;
  const uint32_t b = qy ? (qx ? J.base[3] : J.base[2]) : (qx ? J.base[1] : J.base[0]);
  return b + (uint32_t)(sy >> J.y.parmask) * (uint32_t)(qx ? J.x.width[1] : J.x.width[0]) + (uint32_t)(sx >> J.x.parmask);
}

// Where a sub-cell's count lies.  Four counts a sector would have the adds of
// points in no order wait for one another where the sub-cells are few: a bare
// kernel's read and add for each of 100 M points take 1.21 ms with counts 4
// bytes apart and 0.93 with 16 at 25,600 sub-cells, 0.95 and 0.76 at 100,000,
// 0.76 and 0.73 at 700,000; 0.73 and 0.83 at 3 M, past which the counts would
// leave L2.
constexpr int64_t kGridSpreadMax = (int64_t)1 << 20;
__host__ __device__ __forceinline__ int64_t grid_count_slot(const GridJob& J, uint32_t cell) {
  return (int64_t)cell + 3 * (int64_t)(cell < J.spread ? cell : J.spread);
}

// Number of sub-cells of a job.
inline int64_t grid_cells(const GridJob& j) { return (int64_t)j.x.nclass * j.y.nclass; }

// Host set-up of one axis (edge arrays and ranges excepted): windows of half
// width wsize / 2 at every `step`, cells of half width bsize / 2.
void grid_axis_setup(double lo, double hi, double step, int32_t whalf, int32_t n, int32_t bsize, int32_t nc, bool merged,
                     GridAxis* a);

// How many entries the tables of one cloud take (OWM_ERANGE when its sub-cells
// cannot be numbered in 32 bits), and its job, pointers excepted.
struct GridSizes {
  int64_t nsub = 0, nwin = 0, ncell = 0, rows = 0, edges = 0;
  int64_t main = 0;     // sub-cells that points in no order spread over (the full ones)
  int64_t counts = 0;  // words of the counts
  int64_t chunks = 0;  // of a stage-2 bitmap
  bool merged = false;  // cells share the windows' sub-cells
};
int grid_sizes(const owm_params& p, int64_t n, GridSizes* z);
void grid_job(const owm_params& p, int64_t n, const GridSizes& z, GridJob* j);

// The pieces of the path, in order, on stream s.
struct GridPlan {
  GridJob job;
  GridSizes z;
  int64_t n = 0;
  bool bitmap2 = true;     // stage 2 by occupancy bitmaps (overlap > 0)
  size_t clear_bytes = 0;  // from the scratch's start
  size_t bytes = 0;
  uint32_t *part = nullptr, *llp = nullptr, *s3 = nullptr, *flags = nullptr, *pos = nullptr;
  int64_t* seeds = nullptr;
  void *s2_temp = nullptr, *scan_temp = nullptr;
  size_t s2_bytes = 0, scan_bytes = 0;
  char* base = nullptr;
};
// Sizes the plan (scratch nullptr) or carves it from scratch.  stage1_only: the
// window results alone, in g->job.win.
int grid_plan(const owm_params& p, int64_t n, void* scratch, GridPlan* g, bool stage1_only = false);
// Clears the tables and computes edges and ranges.
int grid_prepare(const GridPlan& g, const owm_params& p, uint32_t* status, cudaStream_t s, int64_t* launches);
// Folds the cloud's points.
int grid_fold(const GridPlan& g, const GridPoints& pts, uint32_t* status, cudaStream_t s, int64_t* launches);
// Stage 1 (rows, windows), stage 2 with stage 3's marks, stage 3 and the seeds.
int grid_windows(const GridPlan& g, cudaStream_t s, int64_t* launches);
int grid_stage2(const GridPlan& g, const owm_params& p, const double* xy, int xy_stride, uint32_t* d_nllp,
                cudaStream_t s, int64_t* launches);
// Where a run's result goes: status, nllp, ns3 are device words; seeds and words
// (ResultBuffer's) may be pinned host memory.
constexpr int kResultStatus = 0, kResultLlp = 3, kResultS3 = 4;  // words, as kStatusSlot, kLlpSlot, kS3Slot
struct GridResult {
  uint32_t *status = nullptr, *nllp = nullptr, *ns3 = nullptr;
  int64_t* seeds = nullptr;
  uint32_t* words = nullptr;
};
// Whether a run takes one launch (grid_small) in place of all of these.
bool grid_is_small(const GridPlan& g);
int grid_small(const GridPlan& g, const owm_params& p, const GridPoints& pts, const double* xy, int xy_stride,
               const GridResult& out, cudaStream_t s, int64_t* launches);
int grid_stage3(const GridPlan& g, const GridResult& out, cudaStream_t s, int64_t* launches);

// Many tiles at once: one launch per step, every tile with its own job.
struct GridBatch {
  int32_t ntiles = 0, chunk = 0;  // chunk: points per fold block
  int32_t bitmap2 = 1;            // every tile has overlap > 0
  int32_t tile_bits = 1, id_bits = 1;
  int64_t items = 0, folds = 0, rows = 0, wins = 0, chunks = 0, cells = 0;  // totals over the tiles
  int64_t row_blocks = 0, win_blocks = 0;  // of 256 rows (windows) of one tile
  size_t clear_bytes = 0, table_bytes = 0, bytes = 0;
  char* base = nullptr;
  char *zid = nullptr, *count = nullptr, *cell_zid = nullptr, *mark = nullptr, *edges = nullptr, *row_mem = nullptr,
       *cellmin = nullptr;
  // device tables, written by the host for each batch: the jobs and, per kind
  // of item, the tiles' first ones
  GridJob* jobs = nullptr;
  int64_t *item_off = nullptr, *fold_off = nullptr, *row_off = nullptr, *win_off = nullptr, *winb_off = nullptr,
          *chunk_off = nullptr,
          *cell_off = nullptr;
  uint32_t *bitmap = nullptr, *part = nullptr, *llp = nullptr, *llp_off = nullptr, *s3cnt = nullptr, *words = nullptr;
  int64_t *out = nullptr, *out_off = nullptr;
  uint32_t *win = nullptr, *k0 = nullptr, *k1 = nullptr, *flags = nullptr, *pos = nullptr, *cnt2 = nullptr;
  void *sort_temp = nullptr, *scan_temp = nullptr;
  size_t sort_bytes = 0, scan_bytes = 0;
};
// Sizes and lays out a batch (base nullptr: sizes only; else 256-byte aligned).
// p[t], n[t]: parameters and points per tile; z[t] gets the tile's sizes.
int grid_batch_plan(const owm_params* p, const int64_t* n, int32_t ntiles, GridSizes* z, char* base, GridBatch* g);
// The tables of a batch that was laid out, as they go to the device: table_bytes
// from g.jobs on.  rec[t]: the tile's points on the device.
void grid_batch_tables(const owm_params* p, const int64_t* n, const GridSizes* z, const double* const* rec, const GridBatch& g,
                       char* host);
// All device work of a batch whose tables are on the device; words[0] is the
// status word.  out and out_off hold the seeds.  Capturable.
int grid_batch_run(const GridBatch& g, cudaStream_t s, int64_t* launches);

}  // namespace owm

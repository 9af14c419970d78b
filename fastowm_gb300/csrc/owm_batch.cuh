// Batched tiles: many independent clouds built and queried together.
#pragma once

#include <string>
#include <vector>

#include "owm_ctx.cuh"

namespace owm {

// Per-tile record read by the batched kernels (all offsets are global).
struct TileMeta {
  int64_t pt_off;   // first point in the concatenated point arrays
  int32_t n;        // points
  int32_t leaf;     // leaf size L (power of two <= 256)
  int32_t leaf_off; // first global leaf
  int32_t nleaves;
  int32_t node_off; // first global node: internal [0, nl-1), leaves [nl-1, 2nl-1)
  int32_t int_off;  // first global internal-node slot
  double mox, moy, mscale;  // Morton domain (square) of the tile
  int64_t mkx0, mky0;       // integer Morton form (mint): cell = (key(v) - k0) >> sh
  int32_t mshx, mshy, mint, mpad;
  double ox, oy;            // float-box origin (bbox corner)
  double min_x, min_y, displace;
  int32_t ncols, nrows, ncg, nrg;
  int32_t whalf, bhalf, bsize;
  uint32_t thr;     // minNumPoints as stage 1 compares it
  int32_t need_dup; // overlap > 0: LLPs are ids occurring >= 2 times
  int32_t pad;
  int64_t win_off, cell_off;
  int32_t ex_off, ey_off, cx_off, cy_off;
  int64_t bm_word;  // first 32-bit word of the tile's stage-2 bitmaps (ids 0..n)
};

// One batch in flight on one stream: device buffers sized for the largest
// batch seen (kept, so trees stay resident until the next batch reuses them),
// pinned host words for the per-tile output offsets, an optional CUDA graph.
struct BatchRun {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  DeviceBuffer mem;
  int64_t* h_off = nullptr;  // pinned [cap_tiles+1] per-tile output offsets, then the status word
  int64_t cap_tiles = 0;
  char* h_stage = nullptr;   // pinned staging of the per-batch tables (copies from it never block)
  size_t stage_cap = 0;
  int64_t launches = 0;
  bool use_graphs = false;
  cudaGraphExec_t graph = nullptr;
  std::string graph_sig;
  int32_t nclass = 0;
  int64_t class_bound[8] = {};
  int32_t class_leaf[8] = {};
  owm_tuning tuning = {4, 4, 256, 0};  // launch shapes (a batch takes its context's)
  // results of the last launch
  int32_t ntiles = 0;
  int64_t total_out = 0;
  int64_t* d_out = nullptr;
  uint32_t* d_status = nullptr;
  size_t bytes_needed = 0;
  cudaEvent_t done = nullptr;
  int init(int device, cudaStream_t s);
  void destroy();
  int leaf_for(int64_t n, int32_t requested) const;
  // Whether these tiles run on the window grid, and the device bytes they take:
  // the grid unless a tile asks for the tree walk, or the grid's tables cannot be
  // numbered or take more than `most` bytes where the trees take less.
  int route(const owm_tile_desc* t, int32_t ntiles, size_t most, bool* grid, size_t* bytes) const;
  // Enqueue everything (copies in, build, stages, offsets out) on `stream`.
  int launch(const owm_tile_desc* t, int32_t ntiles, size_t most = SIZE_MAX);
  int launch_grid(const owm_tile_desc* t, int32_t ntiles, size_t most);  // window grid
  int launch_walk(const owm_tile_desc* t, int32_t ntiles);  // trees, persistent stage-1 walk
  void drop_graph();
  int room(size_t device_bytes, size_t stage_bytes, int32_t ntiles);
  template <class Enqueue>
  int run_or_replay(const std::string& sig, Enqueue enqueue);
  // Wait for the launch and copy the seeds / offsets out.
  int finish(int64_t* seeds, int64_t cap, int64_t* offsets, owm_run_info* info);
  bool ready();
};

}  // namespace owm

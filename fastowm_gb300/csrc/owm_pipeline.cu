// The whole OWM path of one cloud on the device, as the reference application
// runs it per loop iteration (CPP-TBB-CPU/application/owm_optim3.cpp:77-230):
// index, stage 1, sort + stage 2, LLP grid + stage 3, and the result (stage-3
// ids followed by the LLPs).  The index is the window grid (owm_grid.cuh), or
// the tree: with stage1_walk, for stage 3 while a walk limit is set, and where the
// grid's tables do not fit.
// Intermediates never leave the device; the host sees two small count words
// and the final seed list.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstring>

#include "owm_ctx.cuh"
#include "owm_grid.cuh"

namespace owm {

namespace {

__global__ void k_bbox(const double* __restrict__ xyz, int stride, int64_t n, long long* __restrict__ out) {
  long long x0 = 0x7FFFFFFFFFFFFFFFll, y0 = 0x7FFFFFFFFFFFFFFFll;
  long long x1 = (long long)0x8000000000000000ull, y1 = (long long)0x8000000000000000ull;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    long long x = dkey(xyz[stride * i]), y = dkey(xyz[stride * i + 1]);
    x0 = min(x0, x);
    x1 = max(x1, x);
    y0 = min(y0, y);
    y1 = max(y1, y);
  }
  for (int o = 16; o >= 1; o >>= 1) {
    x0 = min(x0, __shfl_xor_sync(0xffffffffu, x0, o));
    x1 = max(x1, __shfl_xor_sync(0xffffffffu, x1, o));
    y0 = min(y0, __shfl_xor_sync(0xffffffffu, y0, o));
    y1 = max(y1, __shfl_xor_sync(0xffffffffu, y1, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(out + 0, x0);
    atomicMin(out + 1, y0);
    atomicMax(out + 2, x1);
    atomicMax(out + 3, y1);
  }
}

// Plain x, y, z points into a cloud's 32-byte records (x, y, z, 0), each
// record written whole (two 16-byte stores), and its x, y array; and back.
__global__ void k_pad_points(const double* __restrict__ src, int64_t n, double* __restrict__ rec,
                             double* __restrict__ xy) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double x = src[3 * i], y = src[3 * i + 1], z = src[3 * i + 2];
    double2* d = reinterpret_cast<double2*>(rec + 4 * i);
    d[0] = make_double2(x, y);
    d[1] = make_double2(z, 0.0);
    reinterpret_cast<double2*>(xy)[i] = make_double2(x, y);
  }
}

__global__ void k_unpad_points(const double* __restrict__ src, int64_t n, double* __restrict__ dst) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double2* r = reinterpret_cast<const double2*>(src + 4 * i);
    const double2 a = r[0], b = r[1];
    dst[3 * i] = a.x;
    dst[3 * i + 1] = a.y;
    dst[3 * i + 2] = b.x;
  }
}

// seeds = s3[0..ns3) ++ llp[0..nllp) as int64 ids (-1 never occurs here).
__global__ void k_assemble(const uint32_t* __restrict__ s3, const uint32_t* __restrict__ ns3,
                           const uint32_t* __restrict__ llp, const uint32_t* __restrict__ nllp, int64_t cap,
                           int64_t* __restrict__ seeds) {
  const int64_t a = *ns3, b = *nllp;
  const int64_t tot = min(a + b, cap);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < tot; i += (int64_t)gridDim.x * blockDim.x)
    seeds[i] = i < a ? (int64_t)s3[i] : (int64_t)llp[i - a];
}

size_t al(size_t b) { return (b + 255) & ~(size_t)255; }

}  // namespace

int clear_status(owm_ctx* c) {
  OWM_CUDA_TRY(cudaMemsetAsync(c->d_small + kStatusSlot, 0, 4, c->stream));
  return OWM_OK;
}

int check_input_status(owm_ctx* c) {
  OWM_CUDA_TRY(cudaMemcpyAsync(c->h_small + kStatusSlot, c->d_small + kStatusSlot, 4, cudaMemcpyDeviceToHost,
                               c->stream));
  OWM_CUDA_TRY(cudaStreamSynchronize(c->stream));
  uint32_t st = c->h_small[kStatusSlot];
  if (st & kStatusNonFinite) return OWM_EINVAL;
  if (st & kStatusWalkBound) return OWM_ETIMEOUT;
  return OWM_OK;
}

int device_bbox(owm_ctx* c, const double* d_xyz, int stride, int64_t n, owm_bbox* out) {
  long long init[4] = {0x7FFFFFFFFFFFFFFFll, 0x7FFFFFFFFFFFFFFFll, (long long)0x8000000000000000ull,
                       (long long)0x8000000000000000ull};
  long long* d = reinterpret_cast<long long*>(c->d_small + kBboxSlot);
  long long* h = reinterpret_cast<long long*>(c->h_small + kBboxSlot);
  std::memcpy(h, init, sizeof(init));
  OWM_CUDA_TRY(cudaMemcpyAsync(d, h, sizeof(init), cudaMemcpyHostToDevice, c->stream));
  int64_t g = std::min<int64_t>((n + 255) / 256, 152 * 8);
  const unsigned gb = (unsigned)std::max<int64_t>(g, 1);
  OWM_LAUNCH("k_bbox", c->stream, k_bbox<<<gb, 256, 0, c->stream>>>(d_xyz, stride, n, d));
  count_launch(&c->launches);
  OWM_CUDA_TRY(cudaMemcpyAsync(h, d, sizeof(init), cudaMemcpyDeviceToHost, c->stream));
  OWM_CUDA_TRY(cudaStreamSynchronize(c->stream));
  out->min_x = dkey_inv(h[0]);
  out->min_y = dkey_inv(h[1]);
  out->max_x = dkey_inv(h[2]);
  out->max_y = dkey_inv(h[3]);
  return OWM_OK;
}

int pad_points(const double* src, int64_t n, double* rec, double* xy, cudaStream_t s, int64_t* launches) {
  const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 152 * 16));
  OWM_LAUNCH("k_pad_points", s, k_pad_points<<<g, 256, 0, s>>>(src, n, rec, xy));
  count_launch(launches);
  OWM_CUDA_TRY(cudaGetLastError());
  return OWM_OK;
}

int unpad_points(const double* src, int64_t n, double* dst, cudaStream_t s, int64_t* launches) {
  const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 152 * 16));
  OWM_LAUNCH("k_unpad_points", s, k_unpad_points<<<g, 256, 0, s>>>(src, n, dst));
  count_launch(launches);
  OWM_CUDA_TRY(cudaGetLastError());
  return OWM_OK;
}

int run_stage1(owm_ctx* c, const TreeStore& t, const owm_params& p, Edge* ex, Edge* ey, uint32_t* d_win) {
  int rc = compute_edges(p, t.ox, t.oy, false, ex, ey, c->stream, &c->launches);
  if (rc) return rc;
  QueryJob j;
  j.tree = t.view(c->walk_limit);
  j.ex = ex;
  j.ey = ey;
  j.ncols = (int32_t)p.ncols;
  j.nrows = (int32_t)p.nrows;
  j.thr = p.min_num_points;
  j.cell_order = 0;
  j.patch_lx = patch_log2(c->tuning.walk_patch_x);
  j.skip = nullptr;
  j.out = d_win;
  j.status = c->d_small + kStatusSlot;
  j.warp_begin = 0;
  return run_query(j, c->d_job, c->stream, &c->launches, "k_query_s1");
}

int ResultBuffer::reserve(int64_t room, cudaStream_t s) {
  if (!words) {
    OWM_CUDA_TRY(cudaMallocHost(&words, 256));
    std::memset(words, 0, 256);
  }
  if (room <= cap) return OWM_OK;
  OWM_CUDA_TRY(cudaStreamSynchronize(s));  // an earlier run may still write there
  if (seeds) cudaFreeHost(seeds);
  seeds = nullptr;
  cap = 0;
  const int64_t want = std::max<int64_t>(room + room / 4, 1 << 16);  // fewer steps for clouds that grow
  if (cudaMallocHost(&seeds, (size_t)want * 8) != cudaSuccess) {
    cudaGetLastError();
    seeds = nullptr;
    return OWM_ENOMEM;
  }
  cap = want;
  return OWM_OK;
}

void ResultBuffer::release() {
  if (seeds) cudaFreeHost(seeds);
  if (words) cudaFreeHost(words);
  seeds = nullptr;
  words = nullptr;
  cap = 0;
}

namespace {
// The whole path on the window grid (owm_grid.cuh): no hierarchy is built.
int run_grid(owm_ctx* c, const PointsView& pts, int64_t n, const owm_params& p, ResultBuffer* rb, int64_t direct_max,
             int64_t** d_seeds) {
  GridPlan g;
  int rc = grid_plan(p, n, nullptr, &g);
  if (!rc) rc = c->scratch.reserve(g.bytes, c->stream);
  if (!rc) rc = grid_plan(p, n, c->scratch.ptr, &g);
  if (rc) return rc;
  cudaStream_t s = c->stream;
  g.job.stamps = reinterpret_cast<unsigned long long*>(c->d_small + kStampSlot);
  GridResult out;
  out.status = c->d_small + kStatusSlot;
  out.nllp = c->d_small + kLlpSlot;
  out.ns3 = c->d_small + kS3Slot;
  const bool direct = g.z.nwin + g.z.ncell + 1 <= direct_max;
  out.seeds = direct ? rb->seeds : g.seeds;
  out.words = rb->words;
  *d_seeds = direct ? nullptr : g.seeds;
  GridPoints gp;
  gp.rec = pts.rec;
  gp.stride = pts.rec_stride;
  OWM_CUDA_TRY(cudaEventRecord(c->ev[0], s));
  if (grid_is_small(g)) return grid_small(g, p, gp, pts.xy, pts.xy_stride, out, s, &c->launches);
  rc = grid_prepare(g, p, out.status, s, &c->launches);
  if (!rc) rc = grid_fold(g, gp, out.status, s, &c->launches);
  if (!rc) rc = grid_windows(g, s, &c->launches);
  if (!rc) rc = grid_stage2(g, p, pts.xy, pts.xy_stride, out.nllp, s, &c->launches);
  if (!rc) rc = grid_stage3(g, out, s, &c->launches);
  return rc;
}
}  // namespace

int run_pipeline_enqueue(owm_ctx* c, const PointsView& pts, int64_t n, const owm_bbox& bb, const owm_run_cfg& cfg,
                         ResultBuffer* rb, int64_t direct_max, owm_params* p_out, int64_t** d_seeds, int64_t* room_out) {
  if (validate_tree_cfg(&cfg.tree) != OWM_OK) return OWM_EINVAL;
  owm_params& p = *p_out;
  int rc = owm_params_compute(&bb, n, cfg.wsize, cfg.overlap, cfg.bsize, &p);
  if (rc) return rc;
  const int64_t room = p.ncells + std::max<int64_t>(p.ngrid, 0) + 1;
  *room_out = room;
  rc = rb->reserve(room <= direct_max ? room : 0, c->stream);
  if (rc) return rc;
  rb->words[8] = 0;
  bool walk1 = cfg.stage1_walk;  // stage 1 walks the tree
  if (!walk1 && c->walk_limit == 0) {
    rc = run_grid(c, pts, n, p, rb, direct_max, d_seeds);
    if (rc != OWM_ENOMEM) return rc;
    walk1 = true;  // no room for the tables, nothing queued: a sparse cloud's trees take less
  }
  const int64_t nc = p.ncells, ng = std::max<int64_t>(p.ngrid, 0);
  rc = tree_alloc(&c->tree, &c->tree_mem, n, cfg.tree, c->stream);
  if (rc) return rc;
  // With a walk limit alone, stage 1 counts on the window grid, which needs no
  // walk: the limit acts on the cells.
  GridPlan g1;
  rc = walk1 ? OWM_OK : grid_plan(p, n, nullptr, &g1, true);
  if (rc) return rc;
  // scratch = [tree build | stage 1's grid | stage 2 | stage 3]
  const size_t bbytes = (tree_scratch_bytes(n) + 255) & ~(size_t)255;
  const size_t tbytes = bbytes + ((g1.bytes + 255) & ~(size_t)255);
  const bool bitmap2 = p.overlap > 0.0;
  const size_t s2bytes = bitmap2 ? stage2_bitmap_scratch_bytes(n) : stage2_scratch_bytes(nc);
  const size_t s2al = (s2bytes + 255) & ~(size_t)255;
  size_t sbytes = tbytes + s2al + stage3_scratch_bytes(ng);
  rc = c->scratch.reserve(sbytes, c->stream);
  if (rc) return rc;
  size_t obytes = 2 * al(65536 * sizeof(Edge)) + 2 * al((size_t)nc * 4) + al((size_t)std::max<int64_t>(ng, 1) * 4) +
                  al((size_t)(nc + ng + 1) * 8) + 1024;
  rc = c->outbuf.reserve(obytes, c->stream);
  if (rc) return rc;
  char* op = static_cast<char*>(c->outbuf.ptr);
  auto take = [&](size_t b) {
    void* q = op;
    op += al(b);
    return q;
  };
  Edge* ex = (Edge*)take(65536 * sizeof(Edge));
  Edge* ey = (Edge*)take(65536 * sizeof(Edge));
  uint32_t* win = (uint32_t*)take((size_t)nc * 4);
  uint32_t* llp = (uint32_t*)take((size_t)nc * 4);
  uint32_t* s3 = (uint32_t*)take((size_t)std::max<int64_t>(ng, 1) * 4);
  int64_t* s64 = (int64_t*)take((size_t)(nc + ng + 1) * 8);
  uint32_t* d_nllp = c->d_small + kLlpSlot;
  uint32_t* d_ns3 = c->d_small + kS3Slot;

  cudaStream_t s = c->stream;
  OWM_CUDA_TRY(cudaEventRecord(c->ev[0], s));
  rc = clear_status(c);
  c->tree.gather_block = c->tuning.gather_block;
  if (!rc)
    rc = build_tree(pts, n, bb, cfg.tree, &c->tree, c->scratch.ptr, bbytes, c->d_small + kStatusSlot, s, &c->launches);
  if (rc) return rc;
  void* s2scratch = static_cast<char*>(c->scratch.ptr) + tbytes;
  void* s3scratch = static_cast<char*>(c->scratch.ptr) + tbytes + s2al;
  const size_t s3cap = c->scratch.cap - tbytes - s2al;
  OWM_CUDA_TRY(cudaEventRecord(c->ev[1], s));
  if (walk1) {
    rc = run_stage1(c, c->tree, p, ex, ey, win);
  } else {
    GridPoints gp;
    gp.rec = pts.rec;
    gp.stride = pts.rec_stride;
    rc = grid_plan(p, n, static_cast<char*>(c->scratch.ptr) + bbytes, &g1, true);
    if (!rc) rc = grid_prepare(g1, p, c->d_small + kStatusSlot, s, &c->launches);
    if (!rc) rc = grid_fold(g1, gp, c->d_small + kStatusSlot, s, &c->launches);
    if (!rc) rc = grid_windows(g1, s, &c->launches);
    win = g1.job.win;
  }
  if (rc) return rc;
  OWM_CUDA_TRY(cudaEventRecord(c->ev[2], s));
  rc = bitmap2 ? run_stage2_bitmap(win, nc, n, p.overlap, llp, d_nllp, s2scratch, s2al, s, &c->launches)
               : run_stage2(win, nc, n, p.overlap, llp, d_nllp, s2scratch, s2al, s, &c->launches);
  if (rc) return rc;
  OWM_CUDA_TRY(cudaEventRecord(c->ev[3], s));
  rc = run_stage3(c->tree.view(c->walk_limit, c->tuning.cell_warps), pts.xy, pts.xy_stride, p, llp, d_nllp, nc, s3, d_ns3,
                  s3scratch, s3cap, c->d_small + kStatusSlot, s, &c->launches);
  if (rc) return rc;
  OWM_CUDA_TRY(cudaEventRecord(c->ev[4], s));
  const unsigned ga = (unsigned)std::min<int64_t>((room + 255) / 256, 152 * 8);
  OWM_LAUNCH("k_assemble", s, k_assemble<<<ga, 256, 0, s>>>(s3, d_ns3, llp, d_nllp, room, s64));
  count_launch(&c->launches);
  OWM_CUDA_TRY(cudaGetLastError());
  OWM_CUDA_TRY(cudaMemcpyAsync(rb->words, c->d_small, 32, cudaMemcpyDeviceToHost, s));
  const bool direct = room <= direct_max;
  if (direct) OWM_CUDA_TRY(cudaMemcpyAsync(rb->seeds, s64, (size_t)room * 8, cudaMemcpyDeviceToHost, s));
  *d_seeds = direct ? nullptr : s64;
  return OWM_OK;
}

int run_pipeline(owm_ctx* c, const PointsView& pts, int64_t n, const owm_bbox& bb, const owm_run_cfg& cfg,
                 int64_t* seeds, int64_t cap, int64_t* n_seeds, owm_run_info* info) {
  owm_params p;
  int64_t* s64 = nullptr;
  int64_t room = 0;
  ResultBuffer& rb = c->result;
  int rc = run_pipeline_enqueue(c, pts, n, bb, cfg, &rb, kDirectSeeds, &p, &s64, &room);
  if (rc) return rc;
  cudaStream_t s = c->stream;
  OWM_CUDA_TRY(cudaEventRecord(c->ev[5], s));
  OWM_CUDA_TRY(cudaStreamSynchronize(s));
  if (rb.words[kStatusSlot] & kStatusNonFinite) return OWM_EINVAL;
  if (rb.words[kStatusSlot] & kStatusWalkBound) return OWM_ETIMEOUT;
  const int64_t nllp = rb.words[kLlpSlot], ns3 = rb.words[kS3Slot];
  const int64_t total = nllp + ns3;
  *n_seeds = total;
  // The run's time ends when the seeds are with the caller.  This copy is timed on
  // the host: an event after it would be waited for (5 us of a 140 us call).
  double ms_copy = 0.0;
  if (total > 0 && total <= cap) {
    if (!s64 && !is_device_ptr(seeds)) {
      std::memcpy(seeds, rb.seeds, (size_t)total * 8);
    } else {
      const auto t0 = std::chrono::steady_clock::now();
      OWM_CUDA_TRY(cudaMemcpyAsync(seeds, s64 ? s64 : rb.seeds, (size_t)total * 8, cudaMemcpyDefault, s));
      OWM_CUDA_TRY(cudaStreamSynchronize(s));
      ms_copy = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }
  }
  if (info) {
    std::memset(info, 0, sizeof(*info));
    info->n_llp = nllp;
    info->n_stage3 = ns3;
    info->n_seeds = total;
    info->params = p;
    if (rb.words[8]) {
      unsigned long long t[kGridStamps];
      std::memcpy(t, rb.words + 16, sizeof(t));
      double* ms[4] = {&info->ms_tree, &info->ms_stage1, &info->ms_stage2, &info->ms_stage3};
      for (int k = 0; k < 4; ++k) *ms[k] = 1e-6 * (double)(t[k + 1] - t[k]);
    } else {
      float a = 0, b = 0, d = 0, e = 0;
      cudaEventElapsedTime(&a, c->ev[0], c->ev[1]);
      cudaEventElapsedTime(&b, c->ev[1], c->ev[2]);
      cudaEventElapsedTime(&d, c->ev[2], c->ev[3]);
      cudaEventElapsedTime(&e, c->ev[3], c->ev[4]);
      info->ms_tree = a;
      info->ms_stage1 = b;
      info->ms_stage2 = d;
      info->ms_stage3 = e;
    }
    float f = 0;
    cudaEventElapsedTime(&f, c->ev[0], c->ev[5]);
    info->ms_total = f + ms_copy;
  }
  return total > cap ? OWM_ERANGE : OWM_OK;
}

}  // namespace owm

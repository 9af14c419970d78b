// Stage 1 by exact window classes: the reference's stage-1 result
// (stage1, CPP-TBB-CPU/src/optim3_func.cpp:541-561: per window the (z, id)-min
// of the points strictly inside and their count, kept when the count reaches
// minNumPoints) computed in O(N + windows) over the tree's sorted points.
//
// The window-class identity is in owm_classes.cuh.  Pipeline:
//   classes_prepare   edge keys per axis, s-range of every window column/row,
//                     class tables (cells of at most half a window step, so a
//                     point's class is one table read and two compares),
//                     counter resets
//   aggregation       per sorted point: its sub-cell; warp match + reduce of
//                     (count, (z, id)-min), then per group one atomic add and
//                     one 128-bit atomic min of the (z, id) pair (ties break
//                     on (z, id)) -- fused into the build's gather for
//                     owm_run, or k_cls_aggregate
//   k_cls_rows        per (window column, sub-cell row): reduce along x
//   k_cls_windows     per window: reduce along y, apply minNumPoints
// All integer: containment is exact by construction, and the search starts
// from the sentinel (z = DBL_MAX, id 0) like the reference, so an empty window
// with minNumPoints == 0 yields id 0.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "owm_classes.cuh"

namespace owm {

bool cls_table_geometry(double lo, double hi, double step, int64_t* k0, int* sh, int32_t* Q) {
  if (!(lo > 0.0) || !(hi >= lo) || !(step > 0.0)) return false;
  int64_t blo, bhi;
  std::memcpy(&blo, &lo, 8);
  std::memcpy(&bhi, &hi, 8);
  if ((blo >> 52) != (bhi >> 52)) return false;
  int e = (int)((blo >> 52) & 0x7FF) - 1023;  // value = 1.m * 2^e, ulp = 2^(e-52)
  double cells = (step * 0.5) / std::ldexp(1.0, e - 52);  // key units in half a step
  if (!(cells >= 2.0)) return false;
  int s = 0;
  while (s < 62 && std::ldexp(1.0, s + 1) <= cells) ++s;
  int64_t q = ((dkey(hi) - dkey(lo)) >> s) + 1;
  if (q > kClsMaxTable) return false;
  *k0 = dkey(lo);
  *sh = s;
  *Q = (int32_t)q;
  return true;
}

}  // namespace owm

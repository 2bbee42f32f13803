// Walk of a range of a grid's nodes as rows and segments of rows, shared by
// the weighted-sum kernels and their launcher (plain C++: it is also compiled
// and checked on the host, at sizes that no test would allocate).
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define TQ_HD __host__ __device__ __forceinline__
#else
#define TQ_HD inline
#endif

namespace tq {

struct RowWalk {
  int64_t start, count;  // nodes of the range, flat indices
  int64_t R;             // nodes per row
  int64_t row0, rows;    // rows the range touches
  int64_t seg, segs;     // nodes per segment, segments per row
  int64_t unit0, units;  // the segments that meet the range, counted from row0's first
};

// Unit u < units of the walk: the segment from node j0 of its row, of whose
// nodes [lo, len) are in the range.
struct RowPart {
  int64_t row;  // counted from row0
  int64_t r0;   // flat index of the row's first node
  int64_t j0;
  int lo, len;
};

// A row can be the whole grid, so the distances between a segment and the
// range are clipped to the segment before they become ints.
TQ_HD RowPart row_part(const RowWalk& w, int64_t u) {
  RowPart p;
  u += w.unit0;
  p.row = w.rows == 1 ? 0 : (w.segs == 1 ? u : u / w.segs);
  p.r0 = (w.row0 + p.row) * w.R;
  p.j0 = (u - p.row * w.segs) * w.seg;
  const int64_t lo = w.start - p.r0 - p.j0;
  const int64_t end = w.start + w.count - p.r0 - p.j0, left = w.R - p.j0;
  int64_t len = left < w.seg ? left : w.seg;
  len = end < len ? end : len;
  p.lo = (int)(lo < 0 ? 0 : (lo < w.seg ? lo : w.seg));
  p.len = (int)(len < 0 ? 0 : len);
  return p;
}

TQ_HD RowWalk make_walk(int64_t start, int64_t count, int64_t R, int64_t seg) {
  RowWalk w;
  w.start = start;
  w.count = count;
  w.R = R;
  w.row0 = start / R;
  w.rows = (start + count - 1) / R - w.row0 + 1;
  w.seg = seg;
  w.segs = (R + seg - 1) / seg;
  // A one-dimensional grid is one row: a range of it is a part of the row's
  // segments, and its units alone are shared out over the warps.  (With the
  // units of the whole row, a range of 1/8 left 7/8 of the warps idle.)
  w.unit0 = (start - w.row0 * R) / seg;
  w.units = (w.rows - 1) * w.segs + (start + count - 1 - (w.row0 + w.rows - 1) * R) / seg + 1 - w.unit0;
  return w;
}

}  // namespace tq

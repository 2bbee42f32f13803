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
};

// Unit u of the walk: the segment from node j0 of its row, of whose nodes
// [lo, len) are in the range (none where lo >= len).
struct RowPart {
  int64_t row;  // counted from row0
  int64_t r0;   // flat index of the row's first node
  int64_t j0;
  int lo, len;
};

TQ_HD int64_t row_units(const RowWalk& w) { return w.rows * w.segs; }

TQ_HD int64_t unit_row(const RowWalk& w, int64_t u) { return w.rows == 1 ? 0 : (w.segs == 1 ? u : u / w.segs); }

// A row can be the whole grid, so the distances between a segment and the
// range are clipped to the segment before they become ints.
TQ_HD RowPart row_part(const RowWalk& w, int64_t u) {
  RowPart p;
  p.row = unit_row(w, u);
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
  return w;
}

}  // namespace tq

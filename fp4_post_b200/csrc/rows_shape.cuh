// Launch shape of the row-major quantizer that feeds registers (quantize_rows_kernel): plain host arithmetic, no CUDA.
#pragma once

#include <stdint.h>

namespace metis {

constexpr int kQuantThreads = 256;
// Per-CTA records that a quantizer's scratch holds (see workspace_records).
constexpr int kMaxRecords = 640;

struct RowsShape {
  int bx;              // threads along a row; kQuantThreads / bx rows per CTA and round
  int64_t gx, gy;      // CTAs along a row, CTAs along the rows (which each of them strides over)
  bool records;        // a record per CTA; false: the running maximum and the error word, zeroed in front of the launch
};

// For [rows, 16 * blocks_per_row] with `resident` CTAs on the device at once; `records`: the scratch has room for them.
static inline RowsShape rows_shape(int64_t rows, int64_t blocks_per_row, int64_t resident, bool records) {
  RowsShape s = {1, 0, 0, records};
  // threads along the row: the power of two that pads the row least (hidden 1536 = 96 blocks runs
  // as 3 x 32, not as 128 with a quarter of the lanes idle); ties go to the wider shape
  while (s.bx < blocks_per_row && s.bx < kQuantThreads) s.bx <<= 1;
  for (int cand = s.bx >> 1; cand >= 32; cand >>= 1)
    if ((blocks_per_row + cand - 1) / cand * cand < (blocks_per_row + s.bx - 1) / s.bx * s.bx) s.bx = cand;
  const int by = kQuantThreads / s.bx;
  s.gx = (blocks_per_row + s.bx - 1) / s.bx;
  s.gy = (rows + by - 1) / by;
  // a row of more than kMaxRecords CTAs (10241 blocks and more, at 16 to 32 of them per CTA) has no room for its records
  if (s.gx > kMaxRecords) s.records = false;
  // four waves of resident CTAs (grid-stride over the rows): whole waves leave no tail
  int64_t cap = resident * 4 / s.gx;
  if (s.records && cap > kMaxRecords / s.gx) cap = kMaxRecords / s.gx;
  if (cap < 1) cap = 1;
  if (s.gy > cap) s.gy = cap;
  if (s.gy > 65535) s.gy = 65535;
  if (s.gy < 1) s.gy = 1;
  return s;
}

}  // namespace metis

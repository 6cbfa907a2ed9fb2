// Launch shapes and rules of the quantizers and the fused norm: plain host arithmetic, no CUDA.
#pragma once

#include <stdint.h>

namespace metis {

constexpr int kQuantThreads = 256;
// Per-CTA records that a quantizer's scratch holds (see workspace_records).
constexpr int kMaxRecords = 640;

// Of the row-major quantizer that feeds registers (quantize_rows_kernel).
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

// CTAs per SM of the tile quantizer for a tensor of `bytes` (whole rows as they lie).  Three fit (~63 KiB each).  Two, or one, where rows do
// not start on 128-byte lines (split_lines) and the tensor is larger than L2: a tile's rows end in the middle of lines that the tile to the
// right begins with, and with more tiles in flight those lines come from memory twice.  The more work there is on a tile (the mean above all,
// stochastic rounding little) the further off the line.  First pass and scale pass, us, bf16 unless stated:
//   three / two CTAs   one output 15568 x 4112 44.6 / 39.6, 21088 x 8304 138 / 98, stochastic 54192 x 8304 424 / 299; centred 23360 x 4112
//                      63.1 / 62.7, 31136 x 4112 86.6 / 81.4, stochastic 30112 x 8304 200 / 143, fp32 30400 x 4112 149 / 114; transposed
//                      15568 x 4112 57.8 / 57.2, 21088 x 8304 189 / 163, centred 31136 x 4112 120 / 106 (but 15424 x 8304 79.4 / 83.0), fp32 and
//                      centred 7712 x 8304 68.7 / 69.2, 15056 x 8304 146 / 132 (but 8736 x 14320 125 / 141); both 15568 x 4112 103 / 95.7,
//                      centred and stochastic 23360 x 4112 113 / 103, 31136 x 4112 230 / 171, fp32 15568 x 4112 132 / 114
//   two / one          both, not centred 42560 x 4112 207 / 193, 21088 x 8304 302 / 218, 54192 x 8304 1011 / 553, fp32 15056 x 8304 251 / 190 (but stochastic
//                      60800 x 4112 267 / 272); centred 60800 x 4112 247 / 321
static inline int tile_ctas_per_sm(int64_t bytes, bool split_lines, bool mean, bool fp32, bool rows_out, bool cols_out) {
  const int64_t mb = split_lines ? bytes / 1000000 : 0;
  const bool both = rows_out && cols_out;
  if (both && !mean && mb >= 350) return 1;
  return mb >= (!mean || both ? 128 : fp32 && cols_out ? 384 : 256) ? 2 : 3;
}

// Fused norm of bf16 rows of 16 bpr elements by a warp per row: the row in shared memory, or in registers.
// Staging rows keeps more warps on an SM, which is what the codes alone of long inputs need; a normalised tensor written beside them, or gamma
// read from global memory in fp32, asks for bandwidth instead, and what staging costs is no longer hidden.  Below 1600 rows staged ones
// go once round, where registers hold too few of them.  Both launches, inputs not in L2, in registers / staged, us (rmsnorm_quant.cu has more):
//   bf16 gamma, codes alone   1300 x 2576 1.05 as fast staged, 2048 x 1552 0.92, 3000 x 2560 0.98, 8192 x 2560 1.01, 65536 x 3584 165 / 137
//   bf16 gamma, norm written  3000 x 2560 12.0 / 12.6, 4096 x 2576 15.7 / 17.4, 16384 x 2048 34.1 / 36.2, 65536 x 2560 146 / 162, 8192 x 3584
//                             33.8 / 35.6, 12000 x 4096 52.8 / 53.7; but 16384 x 1088 23.8 / 22.9, 4096 x 3600 22.1 / 20.6
//   fp32 gamma, codes alone   6000 x 2048 15.4 / 16.8, 12000 x 1552 22.8 / 24.7; but 1300 x 2048 7.9 / 7.5, 4096 x 2576 17.0 / 16.8, and where
//                             rows are fetched swizzled 32768 x 2048 1.05 as fast staged
//   fp32 gamma, norm written  not swizzled 32768 x 2064 121 / 132, 16384 x 4080 125 / 139; but 8192 x 2064 37.2 / 35.8, and swizzled
//                             32768 x 2048 113 / 109
static inline bool norm_rows_staged(int64_t rows, int64_t bpr, bool fp32_gamma, bool norm, bool swizzled) {
  if (bpr <= 32 || (bpr <= 64 && rows < 16384)) return false;
  if (rows < 1600) return true;
  if (fp32_gamma) return norm ? swizzled || rows < 12000 || bpr <= 80 : bpr > 144 || (swizzled && rows >= 16384);
  if (norm) return (bpr <= 72 && rows >= 16384) || rows < (bpr > 224 ? 12000 : bpr > 192 ? 8192 : 0);
  return bpr > 176 || rows >= 3400;
}

}  // namespace metis

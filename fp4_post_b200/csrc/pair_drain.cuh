// How the epilogue of the CTA-pair product drains its two accumulators: constants only, no CUDA.
#pragma once

#include <stdint.h>

namespace metis {

struct PairDrain {
  static constexpr int kChunks = 8;                // 32-column chunks of an accumulator
  static constexpr int kStride = 160;              // the odd tiles' accumulator starts at this column: [160, 256) belong to both
  static constexpr int kShared = 3;                // chunks in that overlap

  // The k-th chunk that warp `part` of the `parts` warps of a lane quarter reads: the shared ones come first.  For the even
  // accumulator [0, 256) they are its last chunks, for the odd one [160, 416) its first ones.
  static constexpr int chunk(int parts, int part, int k, uint32_t odd) {
    return ((odd ? 0 : kChunks - kShared) + part + parts * k) & (kChunks - 1);
  }
  // How many of them it reads in front of its arrival on acc_release.
  static constexpr int before_release(int parts) { return parts == 2 ? 2 : 1; }
  // Arrivals that complete a phase of acc_release: every epilogue warp of both CTAs, whether it reads shared columns or not.
  // The MMAs of tile j wait for the phase of tile j - 1, and they overwrite two things: the columns that the two accumulators
  // share, which the arrivals' own order covers, and all of tile j - 2, which nothing but the arrival of the very warp that read it
  // does (its arrival for tile j - 1 follows its reads of tile j - 2 in program order).  A warp that did not arrive could also fall
  // two phases behind acc_full, whose wait tells parities apart only.
  static constexpr int arrivals(int parts) { return 2 * 4 * parts; }
};

// Epilogue warps per lane quarter of a product [., N] of `stages` pipeline stages a tile, `rounds` tiles a pair, with `vectors` row
// vectors and perhaps an addend C.  Four take half the time for a tile, which is what bounds a product while its epilogue takes
// longer than the MMAs of the next tile, and they end the last tile sooner.  Once the MMAs cover the epilogue, two are faster: what four
// read and store at once takes bandwidth that the operands need, while the next tile starts.  Both sides, us, two / four, L2 cold,
// 14 rounds (8192 x 8192, bf16 D) by stages:
//   nothing        2: 50.1 / 46.0    5: 57.4 / 57.4     6: 62.4 / 66.3     8: 74.6 / 75.9    14: 101.0 / 103.0
//   one vector     6: 72.3 / 65.8    8: 74.7 / 77.8     9: 78.0 / 82.8    16: 109.1 / 114.9
//   two            10: 96.4 / 87.1  14: 104.4 / 104.4  16: 112.9 / 114.9  20: 130.1 / 134.3
//   C              2: 109.7 / 93.0  12: 117.5 / 115.4  16: 127.8 / 131.8  20: 142.2 / 150.8
//   C, one vector  12: 132.1 / 122.9 16: 138.1 / 135.1  20: 148.5 / 153.6
//   C, two         20: 163.9 / 153.7 24: 174.0 / 174.1  32: 218.1 / 228.4
// Fewer rounds weigh the last tile more: 9 stages and a vector 23.5 / 22.6 (2 rounds), 27.6 / 27.5 (3), 36.1 / 36.9 (5), 45.5 / 47.2
// (7); 8 stages 35.7 / 35.0 (5), 50.1 / 50.0 (8); 6 stages and nothing 21.5 / 21.5 (2), 25.6 / 27.6 (3); 16 stages and two vectors
// 44.0 / 42.0 (4), 49.3 / 48.7 (5), 71.8 / 71.7 (8), 20 stages 40.8 / 39.6 (3), 53.9 / 55.3 (5).  Back to back with operands in L2 the
// lines lie a stage lower: a vector and 8 stages 41.6 / 43.0 (8 rounds), two and 14 61.4 / 63.3 (8), C and 14 54.9 / 57.6 (6), C, two and 32
// 60.4 / 63.3 (3).  Stages of the side product count like the others, and an fp32 D has the same lines (both rows of a weight gradient: 16
// stages 133.2 / 136.2, 10 stages 125.1 / 113.6), but its stores and its addend are twice as long: without a vector four gain 1 % at
// most and lose up to 5 (2304 x 4096, 6 stages, 14.8 / 15.6), with C they lose at every length (2 stages 151.6 / 166.8, 16 stages 169.2 /
// 194.6, with a vector 191.5 / 198.6) until two vectors make up for it (12 stages 207.5 / 198.9, 24 227.2 / 226.1, 32 255.0 / 272.3).
// Products of 2018 and 4096 rows have the lines up to two stages lower, and the rule follows them, since the others lose 2 % at most by that: a vector
// and 8 stages 31.6 / 34.2 and 28.0 / 29.5 (5 rounds), 37.5 / 39.0 (7); two vectors and 14 33.9 / 35.1 (4), 38.7 / 39.6 (5); C and 13
// 32.2 / 34.0 (3), 40.5 / 42.7 (4), 60.8 / 62.2 (7), C and 18 26.6 / 29.1 and 25.2 / 26.4 (2); C, a vector and 18 48.2 / 50.8 and 45.3 / 46.1 (4).
// A single column of tiles with chunks outside D gives four warps as many chunks as two have: 1634 x 144 x 1024 5.5 / 5.9, 14842 x 176 x 1280
// with C 9.8 / 10.4; from 200 columns on they are not slower (14842 x 192 x 2304 with a vector 1.02, x 256 1.09 as fast).  One round with an addend alone
// ends with its reads either way (163 x 5296 x 512 7.8 / 8.4, 825 x 416 x 1952 10.9 / 11.3).  300 products drawn from 129 to 16384 rows, 136 to
// 16384 columns and K of 256 to 16384 take 0.96 of their time with two, back to back and L2 cold.
static inline int pair_epilogue_parts(int64_t N, int64_t stages, int64_t rounds, int vectors, bool addend, bool fp32) {
  if (N <= 192 || (fp32 && vectors < (addend ? 2 : 1)) || (addend && vectors == 0 && rounds == 1)) return 2;
  constexpr int kTwoFrom[2][3] = {{6, 8, 14}, {13, 18, 24}};
  const int fewest = addend && vectors == 0 ? 2 : fp32 && vectors == 2 && !addend ? 5 : 3;         // rounds
  return stages >= kTwoFrom[addend][vectors] && rounds >= fewest ? 2 : 4;
}

}  // namespace metis

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

}  // namespace metis

// NVFP4 block quantizer kernels (row-major, transposed and both at once, round-to-nearest and stochastic),
// the scale finalisation pass, column means, and the C entry points that launch them.
//
// The work is split in two launches because of one global dependency: the E4M3 block
// scales are expressed relative to the tensor-wide maximum block scale, while the 4-bit
// codes only depend on their own block.  Pass 1 streams x once, writes the packed codes and
// the fp32 block maxima, and leaves the tensor-wide maximum either in a record per CTA (nothing
// to clear beforehand) or, where the scratch holds no records, in one word by an atomicMax per
// warp.  Pass 2 touches 1/16 of the elements: it turns the block maxima into E4M3 bytes in the
// layout the consumer wants and publishes the per-tensor unit.
#include "common.cuh"
#include "tma.cuh"

#include <atomic>
#include <exception>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>

namespace metis {

constexpr int kHeaderBytes = kWorkspaceHeaderBytes;

__device__ __forceinline__ void fold_global_max(unsigned int* gmax, float local) {
  // amax >= 0, so the IEEE bit pattern orders like the value.
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) local = fmaxf(local, __shfl_xor_sync(0xffffffffu, local, o));
  const unsigned tid = threadIdx.y * blockDim.x + threadIdx.x;
  if ((tid & 31u) == 0 && local > 0.0f) atomicMax(gmax, __float_as_uint(local));
}

// ---- pass 1, row-major ------------------------------------------------------------------------
// One thread owns one 16-element block (two 128-bit loads for bf16): no cross-lane traffic, one
// 64-bit store of codes and one 32-bit store of the block maximum, both coalesced across the warp.
// Thread (tx, ty) of a bx x by CTA walks the rows ty, ty + by*gridDim.y, ... of its fixed column
// block, so there is no division in the loop and the column means stay in registers.
template <typename T, bool kMean, bool kSR>
__global__ void __launch_bounds__(kQuantThreads)
quantize_rows_kernel(const T* __restrict__ x, int rows, int blocks_per_row, int64_t ld,
                     const float* __restrict__ col_mean, const __grid_constant__ PhiloxKeys keys, uint64_t offset,
                     const uint64_t* __restrict__ offset_ctr, uint2* __restrict__ codes, float* __restrict__ amax_out,
                     unsigned int* __restrict__ gmax, unsigned int* __restrict__ records, uint32_t sr16) {
  grid_dependency_wait();
  if (kSR && offset_ctr) offset += *offset_ctr;             // per-device call counter (graph-safe stream of offsets)
  const int bc = blockIdx.x * blockDim.x + threadIdx.x;     // column block of this thread
  const int row_step = gridDim.y * blockDim.y;
  float running = 0.0f;
  if (bc < blocks_per_row) {
    float m[16];
    if (kMean) Load16<float>::load(col_mean + (int64_t)bc * 16, m);
    auto quantize_block = [&](float (&v)[16], int r) {
      if (kMean) subtract16(v, m);
      const float a = abs_max16(v);
      const float s = block_scale_from_amax(a);
      const int64_t b = (int64_t)r * blocks_per_row + bc;
      uint32_t packed[2];
      if (kSR) {
        if (sr16) quantize16_sr(v, s, philox4x32(keys, (uint32_t)b, offset), packed);      // one counter per block
        else quantize16_sr_hw(v, s, philox4x32(keys, (uint32_t)b, offset), packed);
      } else {
        quantize_rn<2>(v, s, packed);
      }
      codes[b] = make_uint2(packed[0], packed[1]);
      amax_out[b] = a;
      running = fmaxf(running, a);
    };
    // the next row's loads are issued before the current block is worked on
    int r = blockIdx.y * blockDim.y + threadIdx.y;
    RawBlock<T> cur, nxt;
    if (r < rows) cur.load(x + (int64_t)r * ld + (int64_t)bc * 16);
    for (; r < rows; r += row_step) {
      const int rn = r + row_step;
      if (rn < rows) nxt.load(x + (int64_t)rn * ld + (int64_t)bc * 16);
      float v[16];
      cur.unpack(v);
      quantize_block(v, r);
      cur = nxt;
    }
  }
  // whole warps reach this point together: a warp never spans the bc bound unevenly in y
  if (!records) {
    fold_global_max(gmax, running);
    return;
  }
  // a record per CTA (see TileOutputs): nobody has to zero a shared maximum first
  __shared__ unsigned int s_max[kQuantThreads / 32];
  const unsigned tid = threadIdx.y * blockDim.x + threadIdx.x;
  const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(running));
  if ((tid & 31u) == 0) s_max[tid >> 5] = m;
  __syncthreads();
  if (tid == 0) {
    unsigned top = 0u;
    for (unsigned w = 0; w < blockDim.x * blockDim.y / 32; ++w) top = max(top, s_max[w]);
    const unsigned cta = blockIdx.y * gridDim.x + blockIdx.x;
    records[3 * cta] = top;
    records[3 * cta + 1] = 0u;
    records[3 * cta + 2] = 0u;
    if (cta == 0) records[-1] = gridDim.x * gridDim.y;
  }
}

// ---- pass 1 on shared-memory tiles: the transposed quantization, alone or together with the row-major one ----
// Output Qt = quantize(x^T): blocks of 16 run along the rows of x.  A persistent CTA walks tiles of
// 128 rows x 128 bytes of x (64 bf16 or 32 fp32 columns) that one thread fetches with TMA (128-byte
// swizzle) into a ring of three stages, two tiles ahead of the arithmetic.
//   column phase  lane w of warp rb reads word w of the 16 rows of row block rb: one (fp32) or two (bf16)
//                 columns of x, i.e. whole blocks of Qt, quantized in registers like a row block.  The 8
//                 code bytes per block are parked in shared memory so that global stores are 64-byte
//                 runs along the token dimension.
//   row phase     (kRowsOut: the "dual" mode) the same tile is read once more along its rows, 16 columns
//                 per thread, and the row-major quantization goes straight to global memory.  The tensor
//                 is read from HBM once for both orientations.
// Both phases read shared memory without bank conflicts thanks to the swizzle (16-byte chunk c of row
// r sits at chunk c ^ (r & 7)).  One __syncthreads per tile: staging and the column means are double
// buffered.  A tile load that does not arrive within the wait limit raises the error word of the
// workspace header (the scale pass then publishes NaN as the unit) instead of hanging.
// What bounds it: instruction issue (24 warps per SM, 63 % of the slots; the rows-only form runs at 86 % of the copy
// bandwidth).  So what stands beside the arithmetic is kept short: a tile that lies inside the tensor has no tests of edges,
// the walk and the block indexes advance by 32-bit additions, the round keys of the random numbers come as parameters, the
// mean is added by the instruction that takes a bf16 operand, shared memory is addressed as such, and the rotation and the
// 16-bit rounding, which training does not ask for, have kernels of their own (kPlain: neither).  Measured at 16384 x 4096
// bf16, this pass alone, rows / transposed / both / both centred and stochastic: 32.9 / 39.6 / 63.8 / 78.6 us before that
// (199 instructions per block in the last one), 30.4 / 33.2 / 55.5 / 60.2 now (150).
template <typename T> struct TileCfg {
  static constexpr int kRows = 128;
  static constexpr int kCols = 128 / sizeof(T);            // 64 (bf16) or 32 (fp32): 128 bytes per row
  static constexpr int kStages = 3;
  static constexpr int kStageBytes = kRows * 128;          // 16 KiB
  static constexpr int kRowBlocks = kRows / 16;            // 8 = warps per CTA
  static constexpr int kColsPerWord = 4 / sizeof(T);       // columns in one 32-bit word of a row: 2 or 1
  static constexpr int kBlocksPerRow = kCols / 16;         // row-phase blocks per tile row: 4 or 2
  static constexpr int kRowUnits = kRows * kBlocksPerRow / kQuantThreads;   // row-phase blocks per thread: 2 or 1
  // staged codes of Qt: per 32-bit word of a row and per column of that word, 64 bytes (128 tokens) at a
  // pitch of 72; the second column's array starts 16 banks off the first
  static constexpr int kCodePitch = 72;
  static constexpr int kCodeArray = 32 * kCodePitch + 64;
  static constexpr int kStagingBytes = kColsPerWord * kCodeArray + kRowBlocks * kCols * 4;
  static constexpr int kSmemBytes = kStages * kStageBytes + 2 * kStagingBytes + 2 * kCols * 4 + 64 + 1024;
};
constexpr int64_t kTileRowsMinElements = 1 << 20;          // row-major tensors from this size on go through the tile kernel
constexpr int64_t kMaxElements = (int64_t)1 << 36;         // blocks are counted in 32 bits (TileWalk, philox4x32)
constexpr uint64_t kColumnStream = 1ull << 63;             // Philox counter space of the transposed output in dual mode

// Workspace of the dual quantizer: word 63 = number of CTA records, records from word 64 on (3 words per CTA),
// then the block maxima of Q and of Qt.
constexpr int kDualMaxCtas = kMaxRecords;
constexpr int kDualHeaderBytes = 256 + ((kDualMaxCtas * 3 * 4 + 255) / 256) * 256;

// How a CTA walks the tiles: their number, those along a row of x, and gridDim.x split into whole rows of tiles
// and a remainder; blocks per row of Q (bpr) and of Qt (bpc), and what a step and the wrap to the next row of tiles add to the index
// of a tile's first block in Q (_r) and in Qt (_t).  Block indexes are counted modulo 2^32 and a tensor has fewer blocks
// (kMaxElements), so the additions end in the right place whichever way they wrap.
struct TileWalk {
  uint32_t tiles, col_tiles, step_rows, step_cols;
  uint32_t bpr, bpc, step_r, wrap_r, step_t, wrap_t;
};

struct TileOutputs {
  uint8_t* codes_t;  float* amax_t;  unsigned int* gmax_t;        // Qt [cols, rows]
  uint8_t* codes_r;  float* amax_r;  unsigned int* gmax_r;        // Q  [rows, cols] (dual mode)
  unsigned int* error;
  // dual mode: instead of folding into the three header words above (which somebody has to zero first), CTA b
  // leaves {largest maximum of Q, of Qt, error} in records[3b..3b+2] and CTA 0 the number of CTAs in records[-1]
  unsigned int* records;
  uint32_t hadamard;         // bit 16: rotate every 16-row block of Qt first; bits [0, 16): the sign of each row
  uint32_t sr16;             // stochastic rounding in software with 16 random bits per element instead of the hardware conversion's 8
};

// y = H (s . v) for one block of 16 values: the signs flip as the mask says, then the 16-point Walsh-Hadamard
// butterfly in natural (Sylvester) order, fp32 additions in this fixed order (bitlinear.py:75-211: the random
// Hadamard transform of the NVIDIA baseline, x -> (x . signs) H per tile of 16, H unnormalised).
__device__ __forceinline__ void hadamard16(float (&v)[16], uint32_t sign_mask) {
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(__float_as_uint(v[i]) ^ (((sign_mask >> i) & 1u) << 31));
#pragma unroll
  for (int h = 1; h < 16; h <<= 1) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if ((i & h) == 0) {
        const float a = v[i], b = v[i + h];
        v[i] = __fadd_rn(a, b);
        v[i + h] = __fsub_rn(a, b);
      }
    }
  }
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(x), "r"(y) : "memory");
}

template <typename T, bool kMean, bool kSR, bool kRowsOut, bool kColsOut, bool kPlain>
__global__ void __launch_bounds__(kQuantThreads, 3)
quantize_tile_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ TileWalk walk, int64_t rows, int64_t cols,
                     const float* __restrict__ col_mean, const __grid_constant__ PhiloxKeys keys, uint64_t offset,
                     const uint64_t* __restrict__ offset_ctr, const __grid_constant__ TileOutputs out) {
  using TC = TileCfg<T>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* s_staging = smem + TC::kStages * TC::kStageBytes;                    // [2][kStagingBytes]
  float* s_mean = reinterpret_cast<float*>(s_staging + 2 * TC::kStagingBytes);  // [2][kCols], negated
  uint64_t* full = reinterpret_cast<uint64_t*>(s_mean + 2 * TC::kCols);         // [kStages]
  __shared__ int s_failed;

  grid_dependency_wait();
  if (kSR && offset_ctr) offset += *offset_ctr;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const uint32_t bpr = walk.bpr, bpc = walk.bpc;
  // Tile id = row tile * col_tiles + column tile; the CTA takes the ids blockIdx.x + i * gridDim.x.  Its coordinates and
  // its first blocks in Q and Qt advance by additions (walk.step_* = gridDim.x in mixed radix): multiplications and 64-bit
  // arithmetic there cost as much as three elements of every tile.
  const uint32_t tiles = walk.tiles, col_tiles = walk.col_tiles;

  if (tid == 0) {
    for (int s = 0; s < TC::kStages; ++s) mbar_init(&full[s], 1);
    s_failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  // -mean of column tile ct's columns, one per thread (added, it rounds as the mean subtracted)
  auto minus_mean = [&](uint32_t ct) {
    const uint32_t c = ct * TC::kCols + tid;
    return kMean && tid < TC::kCols && c < (uint32_t)cols ? -__ldg(col_mean + c) : 0.0f;
  };
  uint32_t rt = blockIdx.x / col_tiles, ct = blockIdx.x - rt * col_tiles;
  uint32_t blk_r = rt * TC::kRows * bpr + ct * TC::kBlocksPerRow, blk_t = ct * TC::kCols * bpc + rt * TC::kRowBlocks;
  if (kMean && tid < TC::kCols) s_mean[tid] = minus_mean(ct);
  __syncthreads();

  uint32_t ahead_rt = rt, ahead_ct = ct, ahead = blockIdx.x;       // the next tile to be requested
  auto issue = [&](int stage) {
    if (ahead < tiles) {
      mbar_expect_tx(&full[stage], TC::kStageBytes);
      tma_load_2d(smem + stage * TC::kStageBytes, &map_x, (int32_t)(ahead_ct * TC::kCols), (int32_t)(ahead_rt * TC::kRows), &full[stage]);
      ahead += gridDim.x;
      ahead_ct += walk.step_cols;
      ahead_rt += walk.step_rows;
      if (ahead_ct >= col_tiles) { ahead_ct -= col_tiles; ++ahead_rt; }
    }
  };
  if (tid == 0) {
    for (int s = 0; s < TC::kStages; ++s) issue(s);
  }

  float running_t = 0.0f, running_r = 0.0f;
  const uint32_t smem_base = smem_u32(smem), staging_base = smem_u32(s_staging), mean_base = smem_u32(s_mean), failed_addr = smem_u32(&s_failed);
  // Where this thread's work lies inside a tile does not change from tile to tile: per tile only the tile's own
  // position is added.
  // column phase: this lane's word of row r of its row block, r = 0..7 (the swizzle repeats from there)
  uint32_t word_at[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) word_at[r] = (uint32_t)(warp * 16 + r) * 128u + ((((uint32_t)lane >> 2) ^ (uint32_t)r) << 4) + ((uint32_t)lane & 3u) * 4u;
  const uint32_t col_blk = (uint32_t)(lane * TC::kColsPerWord) * bpc + warp;    // its first block in Qt
  const uint32_t col_staged = (uint32_t)(lane * TC::kCodePitch + warp * 8);
  // row phase: block (row_r + u * kRowStep, row_b)
  constexpr uint32_t kRowStep = kQuantThreads / TC::kBlocksPerRow;
  const uint32_t row_b = tid & (TC::kBlocksPerRow - 1), row_r = tid / TC::kBlocksPerRow;
  const uint32_t row_blk = row_r * bpr + row_b;
  // write-out of Qt: 8-byte piece out_piece of the out rows out_j, out_j + 32, ...
  const uint32_t out_j = tid >> 3, out_piece = tid & 7;
  const uint32_t out_blk = out_j * bpc + out_piece;
  const uint32_t out_staged = (out_j % TC::kColsPerWord) * TC::kCodeArray + (out_j / TC::kColsPerWord) * TC::kCodePitch + out_piece * 8;
  constexpr uint32_t kAmaxAt = TC::kColsPerWord * TC::kCodeArray;               // staged maxima: [kRowBlocks][kCols]

  // The arithmetic of one tile.  kWhole: all of it lies inside the tensor; the tests of the edges are then not in the code
  // (and the stores of a block not behind a branch).
  auto quantize_tile = [&](auto whole, uint32_t tile_smem, uint32_t staging, uint32_t mean, int live_rows, int live_cols) {
    constexpr bool kWhole = decltype(whole)::value;
    // ---- column phase: warp = row block, lane = 32-bit word of the row ----
    if constexpr (kColsOut) {
      float v[TC::kColsPerWord][16];
      float m[2] = {0.0f, 0.0f};
      if constexpr (kMean) {
        if constexpr (TC::kColsPerWord == 2) { const uint2 both = lds64(mean + lane * 8); m[0] = __uint_as_float(both.x); m[1] = __uint_as_float(both.y); }
        else                                 { m[0] = __uint_as_float(lds32(mean + lane * 4)); }
      }
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const uint32_t w = lds32(tile_smem + word_at[r & 7] + (r >> 3) * 1024);
        if constexpr (sizeof(T) == 4)  { v[0][r] = __uint_as_float(w); }
        else if constexpr (kMean)      { add_bf16x2(w, m[0], m[1], v[0][r], v[1][r]); }
        else                           { v[0][r] = bf16_lo(w); v[1][r] = bf16_hi(w); }
      }
      if constexpr (kMean && sizeof(T) == 4) {
        const f32x2 minus_m = pack2(m[0], m[0]);
#pragma unroll
        for (int r = 0; r < 16; r += 2) split2(add2(pack2(v[0][r], v[0][r + 1]), minus_m), v[0][r], v[0][r + 1]);
      }
      float amax[TC::kColsPerWord];
#pragma unroll
      for (int c = 0; c < TC::kColsPerWord; ++c) {
        if (!kPlain && out.hadamard) hadamard16(v[c], out.hadamard & 0xFFFFu);           // uniform over the grid
        const float a = abs_max16(v[c]);
        const float s = block_scale_from_amax(a);
        uint32_t packed[2];
        if constexpr (kSR) {
          const uint4 bits = philox4x32(keys, blk_t + col_blk + c * bpc, kRowsOut ? (offset ^ kColumnStream) : offset);   // alone: the transposed call's own stream
          if (!kPlain && out.sr16) quantize16_sr(v[c], s, bits, packed);
          else quantize16_sr_hw(v[c], s, bits, packed);
        } else {
          quantize_rn<2>(v[c], s, packed);
        }
        sts64(staging + c * TC::kCodeArray + col_staged, packed[0], packed[1]);
        amax[c] = a;
        if (kWhole || (warp * 16 < live_rows && lane * TC::kColsPerWord + c < live_cols)) running_t = fmaxf(running_t, a);
      }
      const uint32_t at = staging + kAmaxAt + (uint32_t)(warp * TC::kCols + lane * TC::kColsPerWord) * 4u;
      if constexpr (TC::kColsPerWord == 2) sts64(at, __float_as_uint(amax[0]), __float_as_uint(amax[1]));
      else                                 sts32(at, __float_as_uint(amax[0]));
    }

    // ---- row phase: a thread owns blocks (row, b) with b fixed, straight to global memory ----
    if constexpr (kRowsOut) {
      [[maybe_unused]] float mb[16];
      if constexpr (kMean) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint4 f = lds128(mean + row_b * 64 + 16 * i);
          mb[4 * i] = __uint_as_float(f.x); mb[4 * i + 1] = __uint_as_float(f.y); mb[4 * i + 2] = __uint_as_float(f.z); mb[4 * i + 3] = __uint_as_float(f.w);
        }
      }
#pragma unroll
      for (int u = 0; u < TC::kRowUnits; ++u) {
        const uint32_t r = row_r + u * kRowStep;
        const uint32_t row_addr = tile_smem + r * 128u;
        const uint32_t swz = r & 7;
        RawBlock<T> raw;
        if constexpr (sizeof(T) == 2) {
          raw.a = lds128(row_addr + (((2 * row_b) ^ swz) << 4));
          raw.b = lds128(row_addr + (((2 * row_b + 1) ^ swz) << 4));
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint4 w = lds128(row_addr + (((4 * row_b + k) ^ swz) << 4));
            raw.q[k] = make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w));
          }
        }
        float v[16];
        if constexpr (kMean) raw.unpack_plus(mb, v);
        else raw.unpack(v);
        const float a = abs_max16(v);
        const float s = block_scale_from_amax(a);
        const uint32_t blk = blk_r + row_blk + u * (kRowStep * bpr);
        uint32_t packed[2];
        if constexpr (kSR) {
          const uint4 bits = philox4x32(keys, blk, offset);
          if (!kPlain && out.sr16) quantize16_sr(v, s, bits, packed);
          else quantize16_sr_hw(v, s, bits, packed);
        } else {
          quantize_rn<2>(v, s, packed);
        }
        if (kWhole || (row_b * 16 < live_cols && r < live_rows)) {
          reinterpret_cast<uint2*>(out.codes_r)[blk] = make_uint2(packed[0], packed[1]);
          out.amax_r[blk] = a;
          running_r = fmaxf(running_r, a);
        }
      }
    }
  };
  // Write-out of Qt: out row j owns 64 contiguous code bytes and 8 maxima of the tile whose first block in Qt is tile_t.
  auto write_columns = [&](auto whole, uint32_t staging, uint32_t tile_t, int live_rows, int live_cols) {
    constexpr bool kWhole = decltype(whole)::value;
#pragma unroll
    for (int k = 0; k < TC::kCols * 8 / kQuantThreads; ++k) {                   // 8-byte pieces: 8 per out row, 32 rows a trip
      static_assert((kQuantThreads / 8) % TC::kColsPerWord == 0, "the staged array of a thread's pieces does not change");
      if (kWhole || (out_piece * 16 < live_rows && out_j + 32 * k < live_cols))
        reinterpret_cast<uint2*>(out.codes_t)[tile_t + out_blk + 32 * k * bpc] = lds64(staging + out_staged + (32 / TC::kColsPerWord) * TC::kCodePitch * k);
    }
    if (tid < TC::kCols * 2) {
      const uint32_t j = tid & (TC::kCols - 1), h = tid / TC::kCols;            // half h: row blocks 4h .. 4h+3
      if (kWhole || j < live_cols) {
        float* dst = out.amax_t + (tile_t + j * bpc + 4 * h);
        float a4[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) a4[k] = __uint_as_float(lds32(staging + kAmaxAt + ((4 * h + k) * TC::kCols + j) * 4));
        if ((kWhole || live_rows == TC::kRows) && (bpc & 3) == 0) {
          *reinterpret_cast<float4*>(dst) = make_float4(a4[0], a4[1], a4[2], a4[3]);
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) if (kWhole || (4 * h + k) * 16 < live_rows) dst[k] = a4[k];
        }
      }
    }
  };

  volatile int* failed = &s_failed;
  int stage = 0;
  uint32_t it = 0;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++it) {
    const uint32_t buf = it & 1;
    uint32_t next_rt = rt + walk.step_rows, next_ct = ct + walk.step_cols, next_r = blk_r + walk.step_r, next_t = blk_t + walk.step_t;
    if (next_ct >= col_tiles) { next_ct -= col_tiles; ++next_rt; next_r += walk.wrap_r; next_t += walk.wrap_t; }
    const bool more = tile + gridDim.x < tiles;
    const float next_mean = more ? minus_mean(next_ct) : 0.0f;        // on its way while this tile is worked on

    if (!mbar_wait(&full[stage], (it / TC::kStages) & 1u, failed)) *failed = 1;
    if (lds32(failed_addr) != 0) break;               // every thread sees the same outcome of the barrier, or the flag

    const uint32_t row0 = rt * TC::kRows, col0 = ct * TC::kCols;
    const int live_rows = (int)min((int64_t)TC::kRows, rows - row0);            // of this tile
    const int live_cols = (int)min((int64_t)TC::kCols, cols - col0);            // both multiples of 16 where that output exists
    const bool whole = live_rows == TC::kRows && live_cols == TC::kCols;
    const uint32_t tile_smem = smem_base + stage * TC::kStageBytes;
    const uint32_t staging = staging_base + buf * TC::kStagingBytes;
    const uint32_t mean = mean_base + buf * (TC::kCols * 4);
    if (whole) quantize_tile(std::true_type{}, tile_smem, staging, mean, TC::kRows, TC::kCols);
    else       quantize_tile(std::false_type{}, tile_smem, staging, mean, live_rows, live_cols);

    if (kMean && more && tid < TC::kCols) s_mean[(buf ^ 1) * TC::kCols + tid] = next_mean;      // its last readers passed the previous barrier
    __syncthreads();                                   // staging complete; this tile's stage is free
    if (tid == 0) issue(stage);

    if constexpr (kColsOut) {
      if (whole) write_columns(std::true_type{}, staging, blk_t, TC::kRows, TC::kCols);
      else       write_columns(std::false_type{}, staging, blk_t, live_rows, live_cols);
    }
    rt = next_rt;
    ct = next_ct;
    blk_r = next_r;
    blk_t = next_t;
    if (++stage == TC::kStages) stage = 0;
  }
  if (s_failed) {
    // loads of this CTA may still be in flight: give each a bounded chance to land before the CTA leaves
    if (tid == 0) {
      int st = stage;
      for (uint32_t t = blockIdx.x + it * gridDim.x, k = 0; t < tiles && k < TC::kStages; t += gridDim.x, ++k) {
        const uint64_t t0 = global_ns();
        while (!mbar_try(&full[st], ((it + k) / TC::kStages) & 1u) && global_ns() - t0 < kWaitLimitNs) {}
        if (++st == TC::kStages) st = 0;
      }
      if (!out.records) *out.error = 1u;               // error word of the workspace header
    }
  }
  if (out.records) {
    // every CTA writes its record, so nothing needs zeroing and no two CTAs touch the same word
    __shared__ float2 s_max[kQuantThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      running_r = fmaxf(running_r, __shfl_xor_sync(0xffffffffu, running_r, o));
      running_t = fmaxf(running_t, __shfl_xor_sync(0xffffffffu, running_t, o));
    }
    if (lane == 0) s_max[warp] = make_float2(running_r, running_t);
    __syncthreads();
    if (tid == 0) {
      float2 m = s_max[0];
      for (int w = 1; w < kQuantThreads / 32; ++w) { m.x = fmaxf(m.x, s_max[w].x); m.y = fmaxf(m.y, s_max[w].y); }
      unsigned int* rec = out.records + 3 * (int64_t)blockIdx.x;
      rec[0] = __float_as_uint(m.x);
      rec[1] = __float_as_uint(m.y);
      rec[2] = s_failed ? 1u : 0u;
      if (blockIdx.x == 0) out.records[-1] = gridDim.x;
    }
    return;
  }
  if (kColsOut) fold_global_max(out.gmax_t, running_t);
  if (kRowsOut) fold_global_max(out.gmax_r, running_r);
}

// ---- pass 2: block maxima -> E4M3 bytes + unit ------------------------------------------------------
// blockIdx.y picks the job: the dual quantizer finishes both orientations in one launch.  For METIS_SF_MMA the
// walk covers the padded extent and pads with zero bytes.
struct FinalizeJob {
  const float* amax;  const unsigned int* gmax;  const unsigned int* error;
  int64_t R, sf_cols;
  int32_t sf_layout;
  uint8_t* scales;  float* unit;
  int32_t log_tx;             // log2 of the threads along the tiles of a row
  // optional by-product: row_sums[r] = the sum of the quantized values of row r (unit included), from the
  // codes the first pass wrote.  A weight-gradient product needs these sums of its operands when they
  // were centred; here they cost one extra read of codes that are still in L2 instead of a pass of their own.
  const uint2* codes;  float* row_sums;
  // per-CTA records of the dual quantizer (see TileOutputs) in place of gmax / error: word `which` of each is the maximum
  const unsigned int* records;  int32_t which;
};
struct FinalizeJobs { FinalizeJob job[2]; };

// E4M3 bytes of 4 neighbouring blocks from their maxima (quant.py:23): RN_e4m3(RN_fp32(s / unit)), packed conversions.
// The quotient is the correctly rounded one without a division: s times the reciprocal of the unit in two parts (y, the
// correctly rounded one, and what is left of it) lies within one fp32 step of it, and from there one correction by the
// exact remainder rounds correctly (Markstein: y correctly rounded, the quotient within one step).  Four packed
// instructions for two blocks, no branch.  (The product s y alone, with the division itself next to E4M3 ties, was slower
// wherever the largest maximum of a bf16 tensor puts one of its 128 mantissas on a tie, as 19968 does with 117: a warp in
// 512 blocks then meets some, and the scale pass of one output of 65536 x 3584 took 16 or 29 us from tensor to tensor, 16
// now.)  No quotient overflows: unit comes from the largest s.  A NaN (of s or of the unit) is a NaN either way.
struct UnitDivisor { f32x2 minus_unit, y, y_rest; };
__device__ __forceinline__ UnitDivisor unit_divisor(float unit) {
  const float y = __fdiv_rn(1.0f, unit), rest = __fmul_rn(__fmaf_rn(-unit, y, 1.0f), y);
  return {pack2(-unit, -unit), pack2(y, y), pack2(rest, rest)};
}
__device__ __forceinline__ uint32_t scale_bytes4(const float4 a, const UnitDivisor& by) {
  const f32x2 r6 = pack2(0x1.555556p-3f, 0x1.555556p-3f), minus6 = pack2(-6.0f, -6.0f), tiny = pack2(1e-9f, 1e-9f);
  const f32x2 a2[2] = {pack2(a.x, a.y), pack2(a.z, a.w)};
  float q[4];
#pragma unroll
  for (int h = 0; h < 2; ++h) {                            // block_scale_from_amax, two at a time
    const f32x2 sixth = mul2(a2[h], r6);
    const f32x2 s = add2(fma2(fma2(minus6, sixth, a2[h]), r6, sixth), tiny);
    const f32x2 quot = fma2(s, by.y, mul2(s, by.y_rest));
    split2(fma2(fma2(by.minus_unit, quot, s), by.y, quot), q[2 * h], q[2 * h + 1]);
  }
  const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(q[0], q[1]), __NV_SATFINITE, __NV_E4M3);
  const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(q[2], q[3]), __NV_SATFINITE, __NV_E4M3);
  return lo | (hi << 16);
}

// the four E4M3 bytes of a word as floats (exact)
__device__ __forceinline__ void e4m3x4_to_float(uint32_t packed, float (&f)[4]) {
  const __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(packed & 0xFFFFu), __NV_E4M3);
  const __half2_raw hi = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(packed >> 16), __NV_E4M3);
  const float2 l = __half22float2(__half2(lo)), h = __half22float2(__half2(hi));
  f[0] = l.x; f[1] = l.y; f[2] = h.x; f[3] = h.y;
}

// Scale pass of one row: every `step`-th group of four blocks from k on, up to k_live; its bytes go to `to` + k * pitch
// (from there to k_end: zeros, the padding of the tiled layout).  Returns the sum of code x scale.  Not inlined either: the
// loop has four groups in flight and the kernel around it other paths.
__device__ __noinline__ float finish_row(const float* from, const uint2* codes, uint8_t* to, int pitch, int k, int k_live, int k_end,
                                         int step, const UnitDivisor by) {
  float sum = 0.0f;
#pragma unroll 4
  for (; k < k_live; k += step) {
    const float4 a = *reinterpret_cast<const float4*>(from + 4 * (int64_t)k);
    const uint4* w = reinterpret_cast<const uint4*>(codes + 4 * (int64_t)k);
    const uint4 w0 = w[0], w1 = w[1];
    const uint32_t bytes = scale_bytes4(a, by);
    float f[4];
    e4m3x4_to_float(bytes, f);
    sum = fmaf((float)block_code_sum(make_uint2(w0.x, w0.y)), f[0], sum);
    sum = fmaf((float)block_code_sum(make_uint2(w0.z, w0.w)), f[1], sum);
    sum = fmaf((float)block_code_sum(make_uint2(w1.x, w1.y)), f[2], sum);
    sum = fmaf((float)block_code_sum(make_uint2(w1.z, w1.w)), f[3], sum);
    *reinterpret_cast<uint32_t*>(to + (int64_t)k * pitch) = bytes;
  }
  for (; k < k_end; k += step) *reinterpret_cast<uint32_t*>(to + (int64_t)k * pitch) = 0u;
  return sum;
}

// Scale pass of four blocks of each of four rows (row_pitch floats apart) of which only the first `rows` and `blocks` exist, or
// which no vector load reaches: `dst` gets a 16-byte piece of the tiled layout, or single bytes of the rows.  All maxima are
// in flight at once: one after the other they make a chain of sixteen loads at the end of a small tensor.
__device__ __noinline__ void finish_edge(const float* from, int64_t row_pitch, int rows, int blocks, uint8_t* dst, bool tiled, const UnitDivisor by) {
  float a[4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
#pragma unroll
    for (int j = 0; j < 4; ++j) a[c][j] = c < rows && j < blocks ? from[c * row_pitch + j] : 0.0f;
  }
  uint32_t out[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    out[c] = 0u;
    if (c >= rows || blocks <= 0) continue;
    out[c] = scale_bytes4(make_float4(a[c][0], a[c][1], a[c][2], a[c][3]), by);
    if (blocks < 4) out[c] &= (1u << (8 * blocks)) - 1u;
    if (!tiled) {
#pragma unroll
      for (int j = 0; j < 4; ++j) if (j < blocks) dst[c * row_pitch + j] = (uint8_t)(out[c] >> (8 * j));
    }
  }
  if (tiled) *reinterpret_cast<uint4*>(dst) = make_uint4(out[0], out[1], out[2], out[3]);
}

// A thread finishes one 16-byte piece of the tiled layout at a time: the scales of the rows l, l + 32, l + 64, l + 96 of
// a 128-row block for 4 scale columns, i.e. four 16-byte reads of maxima and one 16-byte store (row-major scales: four
// words of four rows).  Two neighbouring lanes take two neighbouring l, the next ones the tiles to the right, so a warp
// reads runs of up to 256 bytes and stores whole 32-byte sectors.  An item is such a pair of l (8 rows) over a segment of
// the row (the whole of it where its sum is wanted); a CTA takes 64 / tx items at once.
// Bound by issue: edges, padding and divisions stay out of the unrolled path (62 instructions per block with them and with
// scalar arithmetic, 27 with packed arithmetic alone).  One output / both / both with token sums, us: 16384 x 4096
// 11.2 / 21.0 / 28.2 before that, 6.6 / 10.4 / 19.7 now; 65536 x 4096 32 / 62 / 79 and 17 / 30 / 67 (the bytes alone take
// 13 / 26 / 46); 64 x 18944, one output, 4.0 and 2.8.
constexpr int kFinThreads = 128;
// What the jobs of a launch want: no row sums, every row made of whole groups of four blocks; no row sums; sums, four rows to
// a thread; sums, up to a CTA to a row (finalize_form has the rule).  Kernels of their own: what stands beside the unrolled
// path costs it 1 % (a call for the edges) to 15 %.
enum FinalizeForm { kFinPlain, kFinEdges, kFinSums, kFinSumsByRow };
// The rows of a job with sums, 2^log_tx threads (up to the whole CTA) to each.
__device__ __forceinline__ void finish_rows(const FinalizeJob& J, bool tiled, int tiles, int groups, float unit, const UnitDivisor& by,
                                            float (&s_sum)[kFinThreads / 32][2][4]) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = 1 << J.log_tx, per_cta = kFinThreads >> J.log_tx;
  const int k_lane = tid & (tx - 1), sub = tid >> J.log_tx;
  const int64_t out_rows = tiled ? (J.R + 127) / 128 * 128 : J.R;                   // whole tiles: zeros behind the last row
  for (int64_t first = (int64_t)blockIdx.x * per_cta; first < out_rows; first += (int64_t)gridDim.x * per_cta) {
    const int64_t r = first + sub;
    float sum = 0.0f;
    if (r < out_rows) {
      uint8_t* to = tiled ? J.scales + (r >> 7) * tiles * 512 + (r & 31) * 16 + ((r >> 5) & 3) * 4 : J.scales + r * J.sf_cols;
      sum = finish_row(J.amax + r * J.sf_cols, J.codes + r * J.sf_cols, to, tiled ? 512 : 4, k_lane, r < J.R ? (int)(J.sf_cols >> 2) : 0,
                       tiled ? groups : 0, tx, by);
    }
    // fixed order: lanes of a row by butterfly, then its warps one after the other
    for (int o = (tx < 32 ? tx : 32) >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (tx > 32) {
      __syncthreads();                                         // the previous round's sums have been read
      if (lane == 0) s_sum[warp][0][0] = sum;
      __syncthreads();
      if (k_lane == 0) for (int w = 1; w < tx >> 5; ++w) sum += s_sum[warp + w][0][0];
    }
    if (k_lane == 0 && r < J.R) J.row_sums[r] = sum * (0.5f * unit);
  }
}

template <FinalizeForm kForm>
__device__ __forceinline__ void finalize_scales(const FinalizeJob& job0, const FinalizeJob& job1, uint64_t* __restrict__ offset_ctr) {
  constexpr bool kSums = kForm == kFinSums || kForm == kFinSumsByRow, kQuadSums = kForm == kFinSums;
  __shared__ unsigned int s_top[kFinThreads / 32], s_bad[kFinThreads / 32];
  __shared__ float s_sum[kFinThreads / 32][2][4];
  grid_dependency_wait();
  const FinalizeJob& J = blockIdx.y == 0 ? job0 : job1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned int top = 0u, bad = 0u;                 // bits of the largest block maximum (>= 0: they order like the value)
  if (J.records) {
    const int n = (int)J.records[-1];
    for (int i = tid; i < n; i += kFinThreads) {
      top = max(top, J.records[3 * i + J.which]);
      bad |= J.records[3 * i + 2];
    }
    top = __reduce_max_sync(0xffffffffu, top);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if (lane == 0) { s_top[warp] = top; s_bad[warp] = bad; }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kFinThreads / 32; ++w) { top = max(top, s_top[w]); bad |= s_bad[w]; }
  } else {
    top = *J.gmax;
    bad = *J.error;
  }
  const float smax = block_scale_from_amax(__uint_as_float(top));
  // quant.py:21-22; a pass-1 kernel that gave up on a load raises the error word: publish NaN so that it shows
  const float unit = bad ? __uint_as_float(0x7FC00000u) : __fdiv_rn(smax, 448.0f);
  if (blockIdx.x == 0 && tid == 0) {
    *J.unit = unit;
    if (offset_ctr && blockIdx.y == 0) *offset_ctr += 1;       // pass 1 of this call has finished: the next call draws fresh bits
  }
  const UnitDivisor by = unit_divisor(unit);

  const bool tiled = J.sf_layout == METIS_SF_MMA;
  const int64_t R = J.R, sf_cols = J.sf_cols;
  const int tiles = (int)sf_tiles_per_row(sf_cols * 16);       // padded to whole stages (METIS_SF_MMA)
  const int groups = tiled ? tiles : (int)((sf_cols + 3) >> 2);
  const bool vec = (sf_cols & 3) == 0;
  const bool sums = kSums && J.row_sums != nullptr;              // the host asks for them only when vec holds
  if constexpr (kForm == kFinSumsByRow) {
    if (sums) {
      finish_rows(J, tiled, tiles, groups, unit, by, s_sum);
      return;
    }
  }
  const int tx = 1 << J.log_tx, per_cta = 64 >> J.log_tx;        // threads along a row, items per CTA
  const int k_lane = (tid >> 1) & (tx - 1), sub = tid >> (1 + J.log_tx);
  const int64_t items = ((R + 127) / 128) * 16;
  // without row sums a row is cut into segments of tx tiles, so that a few wide rows still fill the SMs
  const int segments = sums ? 1 : (groups + tx - 1) >> J.log_tx;
  const int64_t work = items * segments;
  const int64_t row_pitch = 32 * sf_cols;                        // between a thread's four rows
  // the item loop is uniform over the CTA (the sums of a row meet at a barrier)
  for (int64_t first = (int64_t)blockIdx.x * per_cta; first < work; first += (int64_t)gridDim.x * per_cta) {
    const bool live = first + sub < work;
    const int64_t item = segments == 1 ? first + sub : (first + sub) / segments;
    const int k_first = segments == 1 ? 0 : (int)((first + sub) - item * segments) << J.log_tx;
    const int k_end = segments == 1 ? groups : min(groups, k_first + tx);
    const int64_t row0 = (item >> 4) * 128 + (item & 15) * 2 + (tid & 1);       // this thread's rows: row0 + 32 c
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    const float* src = J.amax + row0 * sf_cols;
    const uint2* codes = J.codes + row0 * sf_cols;
    uint8_t* dst = tiled ? J.scales + (item >> 4) * tiles * 512 + ((item & 15) * 2 + (tid & 1)) * 16 : J.scales + row0 * sf_cols;
    const int rows = row0 >= R ? 0 : (int)min((int64_t)4, (R - row0 + 31) >> 5);      // of this thread's four: the first ones
    // the piece of tile k (all four blocks of it exist); kWhole: of four rows, else of the first `rows`
    auto piece = [&](auto whole, int k) {
      constexpr bool kWhole = decltype(whole)::value;
      float4 a[4];
      uint4 cd[4][2];
      uint32_t out[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {                             // every load before the first use
        const float* from = src + c * row_pitch + 4 * k;
        a[c] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (kWhole || c < rows) {
          if (vec) a[c] = *reinterpret_cast<const float4*>(from);
          else     a[c] = make_float4(from[0], from[1], from[2], from[3]);
        }
      }
      if (kQuadSums && sums) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          cd[c][0] = cd[c][1] = make_uint4(0u, 0u, 0u, 0u);
          if (!kWhole && c >= rows) continue;
          const uint4* w = reinterpret_cast<const uint4*>(codes + c * row_pitch + 4 * k);
          cd[c][0] = w[0];
          cd[c][1] = w[1];
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) out[c] = kWhole || c < rows ? scale_bytes4(a[c], by) : 0u;      // 0: padding
      if (kQuadSums && sums) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float f[4];
          e4m3x4_to_float(out[c], f);
          acc[c] = fmaf((float)block_code_sum(make_uint2(cd[c][0].x, cd[c][0].y)), f[0], acc[c]);
          acc[c] = fmaf((float)block_code_sum(make_uint2(cd[c][0].z, cd[c][0].w)), f[1], acc[c]);
          acc[c] = fmaf((float)block_code_sum(make_uint2(cd[c][1].x, cd[c][1].y)), f[2], acc[c]);
          acc[c] = fmaf((float)block_code_sum(make_uint2(cd[c][1].z, cd[c][1].w)), f[3], acc[c]);
        }
      }
      if (tiled) {
        *reinterpret_cast<uint4*>(dst + (int64_t)k * 512) = make_uint4(out[0], out[1], out[2], out[3]);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) if (kWhole || c < rows) *reinterpret_cast<uint32_t*>(dst + c * row_pitch + 4 * k) = out[c];
      }
    };
    for (int k = k_first + k_lane; live && k < k_end; k += tx) {
      const bool full = (vec || tiled) && 4 * k + 4 <= sf_cols;
      if (full && rows == 4) {
        piece(std::true_type{}, k);
      } else if (!kQuadSums && full) {                              // decode: fewer than 128 rows
        piece(std::false_type{}, k);
      } else if constexpr (kForm == kFinPlain) {                    // what is left then is padding
        if (tiled) *reinterpret_cast<uint4*>(dst + (int64_t)k * 512) = make_uint4(0u, 0u, 0u, 0u);
      } else if constexpr (!kQuadSums) {                            // an edge of the tensor, or padding
        const int blocks = (int)(sf_cols - 4 * k < 4 ? sf_cols - 4 * k : 4);
        finish_edge(src + 4 * k, row_pitch, rows, blocks, dst + (tiled ? (int64_t)k * 512 : (int64_t)4 * k), tiled, by);
      } else {                                                      // the same with sums: kept short
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          const int64_t r = row0 + 32 * c;
          uint32_t word = 0u;
          if (r < R) {
#pragma unroll 1
            for (int j = 0; j < 4 && 4 * (int64_t)k + j < sf_cols; ++j) {
              const int64_t b = r * sf_cols + 4 * k + j;
              const uint8_t byte = float_to_e4m3(__fdiv_rn(block_scale_from_amax(J.amax[b]), unit));
              word |= (uint32_t)byte << (8 * j);
              if (!tiled) J.scales[b] = byte;
              if (sums) {
                const float part = (float)block_code_sum(J.codes[b]) * e4m3_to_float(byte);
                if (c == 0) acc[0] += part; else if (c == 1) acc[1] += part; else if (c == 2) acc[2] += part; else acc[3] += part;
              }
            }
          }
          if (tiled) *reinterpret_cast<uint32_t*>(dst + (int64_t)k * 512 + 4 * c) = word;
        }
      }
    }
    if (sums) {
      // fixed order: lanes of an item by butterfly, then its warps one after the other
      for (int o = tx < 16 ? tx : 16; o >= 2; o >>= 1) {
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
      }
      if (tx > 16) {
        if (lane < 2) {
#pragma unroll
          for (int c = 0; c < 4; ++c) s_sum[warp][lane][c] = acc[c];
        }
        __syncthreads();
        const int warps = tx >> 4;                              // per item
        if (k_lane == 0) {
          for (int w = 1; w < warps; ++w) {
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[c] += s_sum[warp + w][tid & 1][c];
          }
        }
        __syncthreads();
      }
      if (live && k_lane == 0) {
        const float half_unit = 0.5f * unit;
#pragma unroll
        for (int c = 0; c < 4; ++c) if (row0 + 32 * c < R) J.row_sums[row0 + 32 * c] = acc[c] * half_unit;
      }
    }
  }
}
// Resident at once: 8 CTAs per SM, 5 and 7 with sums.  The kernel with sums by four rows is left to the compiler (96 registers): asked for its five
// CTAs it is scheduled worse (16384 x 4096, dual quantizer with sums: 92.4 us against 89.9).
template <FinalizeForm kForm>
__global__ void __launch_bounds__(kFinThreads, kForm == kFinSumsByRow ? 7 : 8)
finalize_scales_kernel(const FinalizeJob job0, const FinalizeJob job1, uint64_t* __restrict__ offset_ctr) {
  finalize_scales<kForm>(job0, job1, offset_ctr);
}
__global__ void __launch_bounds__(kFinThreads)
finalize_scales_sums_kernel(const FinalizeJob job0, const FinalizeJob job1, uint64_t* __restrict__ offset_ctr) {
  finalize_scales<kFinSums>(job0, job1, offset_ctr);
}

// ---- small tensors (decode-sized activations): one launch --------------------------------------------------
// Up to 16384 blocks (256 Ki elements), round to nearest.  One thread-block cluster of up to 8 CTAs
// holds the whole tensor: a thread quantizes up to 4 blocks and keeps their maxima in registers, the
// tensor-wide maximum goes through the cluster's shared memory (hardware cluster barrier: nothing to
// zero, no spinning, no scratch in global memory), and the same thread then writes its E4M3 bytes.
// Replaces pass 1 + scale pass of the streaming path (and the zero-fill in front of them where the
// scratch holds no records) where launch latency is all there is to save; with more blocks (or more padding words to clear) the 8 SMs of a cluster lose to the
// streaming kernels on 148.  Measured back to back inside a CUDA graph: 16 x 4096 bf16 4.3 us against
// 8.0, 32 x 4096 5.2, 64 x 4096 6.8 against 8.1.
constexpr int kSmallThreads = 512;
constexpr int kSmallBlocks = 4;                    // blocks per thread
// Blocks up to which the cluster is taken although the streaming path needs no zero-fill either.  8 CTAs of 512 threads: a
// round is 4096 blocks and costs 0.75 us for bf16, 1.1 for fp32, where the two launches stay at 3.7 to 5.5 (a few blocks more
// than whole rounds cost nothing).  Row-major scales, without padding to clear: three rounds for bf16, two for fp32.  Tiled ones:
// one, and a second for bf16 rows of up to 1024 elements.  Cluster / two launches back to back, us: bf16 row-major 64 x 1040
// 3.2 / 4.4, 48 x 4096 4.2 / 4.5, 56 x 4096 4.7 / 4.1, tiled 16 x 4112 3.7 / 4.6, 200 x 528 4.2 / 6.5, 64 x 1536 4.2 / 3.7, 40 x 4096
// 4.9 / 4.5; fp32 row-major 32 x 4112 4.4 / 4.7, 100 x 1536 5.1 / 4.0, tiled 16 x 4112 4.0 / 4.6, 24 x 4096 4.9 / 4.2.  In a chain of
// decode layers, where eight free SMs next to each other have to be found beside the vector products, 20 x 4096 takes
// 21.3 / 20.9 per layer and 24 x 4096 22.2 / 21.7; a single layer of 16 x 8192 35 / 29.
static int64_t cluster_blocks(int64_t C, int32_t sf_layout, int64_t element_bytes) {
  const bool bf16 = element_bytes == 2, narrow = C <= 1024;
  const int rounds = sf_layout == METIS_SF_ROWMAJOR ? (bf16 ? 3 : 2) : (bf16 && narrow ? 2 : 1);
  return (int64_t)rounds * kSmallCtas * kSmallThreads + 64;
}
constexpr int64_t kSmallMaxBlocks = (int64_t)kSmallCtas * kSmallThreads * kSmallBlocks;

template <typename T, bool kMean>
__global__ void __launch_bounds__(kSmallThreads)
quantize_small_kernel(const T* __restrict__ x, int rows, int blocks_per_row, int64_t ld,
                      const float* __restrict__ col_mean, uint2* __restrict__ codes, int32_t sf_layout,
                      int tiles, int padded_words, uint8_t* __restrict__ scales, float* __restrict__ unit_out) {
  __shared__ ClusterMaxSmem s_max;
  grid_dependency_wait();
  const int t = (int)(cluster_cta_rank() * blockDim.x + threadIdx.x);       // CTAs of 32..512 threads: one block per thread while that fits
  const int stride = (int)(cluster_cta_count() * blockDim.x);
  const int real_blocks = rows * blocks_per_row;
  if (sf_layout == METIS_SF_MMA) zero_scale_padding(scales, rows, blocks_per_row, tiles, padded_words, t, stride);

  float amax[kSmallBlocks];
  float running = 0.0f;
  RawBlock<T> raw[kSmallBlocks];
#pragma unroll
  for (int j = 0; j < kSmallBlocks; ++j) {        // all loads first: one trip to memory
    const int b = t + j * stride;
    if (b < real_blocks) {
      const int r = b / blocks_per_row, c = b - r * blocks_per_row;
      raw[j].load(x + (int64_t)r * ld + (int64_t)c * 16);
    }
  }
#pragma unroll
  for (int j = 0; j < kSmallBlocks; ++j) {
    const int b = t + j * stride;
    amax[j] = 0.0f;
    if (b < real_blocks) {
      float v[16];
      raw[j].unpack(v);
      if (kMean) {
        const int r = b / blocks_per_row, c = b - r * blocks_per_row;
        float m[16];
        Load16<float>::load(col_mean + (int64_t)c * 16, m);
        subtract16(v, m);
      }
      const float a = abs_max16(v);
      uint32_t pk[2];
      quantize_rn<2>(v, block_scale_from_amax(a), pk);
      codes[b] = make_uint2(pk[0], pk[1]);
      amax[j] = a;
      running = fmaxf(running, a);
    }
  }

  const float unit = __fdiv_rn(block_scale_from_amax(cluster_fmax(running, s_max)), 448.0f);       // quant.py:21-22
  if (t == 0) *unit_out = unit;

#pragma unroll
  for (int j = 0; j < kSmallBlocks; ++j) {
    const int b = t + j * stride;
    if (b >= real_blocks) continue;
    const int r = b / blocks_per_row, c = b - r * blocks_per_row;
    const float ratio = __fdiv_rn(block_scale_from_amax(amax[j]), unit);      // quant.py:23
    const int64_t off = (sf_layout == METIS_SF_MMA) ? sf_mma_offset(r, c, tiles) : (int64_t)b;
    scales[off] = float_to_e4m3(ratio);             // 4 neighbouring lanes fill one 32-bit word
  }
  cluster_leave();
}

// Whether the one-launch kernel takes a row-major quantization of [R, C].
static bool small_path(int64_t R, int64_t C, int32_t sf_layout, int64_t* tiles, int64_t* padded_words) {
  *tiles = sf_tiles_per_row(C);
  *padded_words = sf_layout == METIS_SF_MMA ? ceil_div(R, 128) * 128 * *tiles : 0;
  return R * (C / 16) <= kSmallMaxBlocks && *padded_words <= kSmallMaxPaddedWords;
}

template <typename T>
static int32_t launch_small(const T* x, int64_t rows, int64_t cols, int64_t ld, const float* mean, uint8_t* codes,
                            int32_t sf_layout, int64_t tiles, int64_t padded_words, uint8_t* scales,
                            float* unit, cudaStream_t st) {
  const int64_t blocks = rows * (cols / 16);
  const int64_t work = blocks > padded_words / 4 ? blocks : padded_words / 4;   // a block, or a 16-byte piece of padding, per thread
  int64_t ctas = ceil_div(work, 32);
  if (ctas > kSmallCtas) ctas = kSmallCtas;
  int64_t threads = ceil_div(ceil_div(work, ctas), 32) * 32;            // spread thin: latency is what counts here
  if (threads > kSmallThreads) threads = kSmallThreads;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = launch_overlap_enabled(kLaunchShort) ? 2 : 1;
  uint2* c2 = reinterpret_cast<uint2*>(codes);
  if (mean)
    METIS_CUDA_OK(cudaLaunchKernelEx(&cfg, quantize_small_kernel<T, true>, x, (int)rows, (int)(cols / 16), ld, mean, c2, sf_layout,
                                     (int)tiles, (int)padded_words, scales, unit));
  else
    METIS_CUDA_OK(cudaLaunchKernelEx(&cfg, quantize_small_kernel<T, false>, x, (int)rows, (int)(cols / 16), ld, mean, c2, sf_layout,
                                     (int)tiles, (int)padded_words, scales, unit));
  return METIS_OK;
}

// ---- column means -----------------------------------------------------------------------------------------
// Stage 1: CTA (bx, by) sums rows [by*rows_per_split, ...) of 8*32 columns into
// partial[by][col]; stage 2 adds the partials in a fixed order and divides by rows.
constexpr int kMeanThreads = 256;
template <typename T>
__global__ void __launch_bounds__(kMeanThreads)
col_partial_sum_kernel(const T* __restrict__ x, int64_t rows, int64_t cols, int64_t ld,
                       int64_t rows_per_split, float* __restrict__ partial, int64_t mean_of_rows) {
  // mean_of_rows > 0 (a single split): `partial` is the mean itself, sum / mean_of_rows, as stage 2 would write it
  grid_dependency_wait();
  // stage 2 follows in the stream: its few CTAs may take their places now (they wait for this grid to complete)
  if (mean_of_rows == 0) grid_launch_dependents();
  // 32 lanes x 8 columns = 256 columns per CTA; 8 warps stride over the rows.
  __shared__ float s_part[kMeanThreads / 32][256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t col = (int64_t)blockIdx.x * 256 + lane * 8;
  const int64_t r_begin = (int64_t)blockIdx.y * rows_per_split;
  const int64_t r_end = min(rows, r_begin + rows_per_split);
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (col < cols) {
    // four rows in flight per warp; the additions keep their order (row after row)
    int64_t r = r_begin + warp;
    for (; r + 3 * (kMeanThreads / 32) < r_end; r += 4 * (kMeanThreads / 32)) {
      float v[4][8];
#pragma unroll
      for (int k = 0; k < 4; ++k) Load8<T>::load(x + (r + k * (kMeanThreads / 32)) * ld + col, v[k]);
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += v[k][i];
    }
    for (; r < r_end; r += kMeanThreads / 32) {
      float v[8];
      Load8<T>::load(x + r * ld + col, v);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += v[i];
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) s_part[warp][lane * 8 + i] = acc[i];
  __syncthreads();
  const int c = threadIdx.x;
  float sum = 0.0f;
#pragma unroll
  for (int w = 0; w < kMeanThreads / 32; ++w) sum += s_part[w][c];
  const int64_t oc = (int64_t)blockIdx.x * 256 + c;
  if (oc < cols) partial[(int64_t)blockIdx.y * cols + oc] = mean_of_rows > 0 ? __fdiv_rn(__fadd_rn(0.0f, sum), (float)mean_of_rows) : sum;
}

constexpr int kMeanMaxSplits = 64;
__global__ void __launch_bounds__(256) col_mean_finish_kernel(const float* __restrict__ partial, int64_t splits, int64_t rows,
                                       int64_t cols, float* __restrict__ mean) {
  grid_dependency_wait();
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  // all loads in flight at once (splits <= kMeanMaxSplits), then the additions in their fixed order
  float v[kMeanMaxSplits];
#pragma unroll
  for (int s = 0; s < kMeanMaxSplits; ++s) v[s] = s < splits ? partial[s * cols + c] : 0.0f;
  float sum = 0.0f;
#pragma unroll
  for (int s = 0; s < kMeanMaxSplits; ++s)
    if (s < splits) sum += v[s];
  mean[c] = __fdiv_rn(sum, (float)rows);
}

static int64_t col_mean_splits(int64_t rows) {
  int64_t s = ceil_div(rows, 128);
  return s < 1 ? 1 : (s > kMeanMaxSplits ? kMeanMaxSplits : s);
}

// ---- launch helpers ------------------------------------------------------------------------------------------

int device_sm_count() {
  static std::atomic<int> known[64] = {};                // by device; 0: not asked yet
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  const bool keep = dev >= 0 && dev < 64;
  if (keep && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
  if (keep) known[dev].store(n, std::memory_order_relaxed);
  return n;
}
int resident_ctas(const void* kernel, int threads, size_t smem) {
  static std::mutex mutex;
  static std::map<std::tuple<const void*, int, size_t, int>, int> known;
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  // nothing may be thrown through the C entry points: without a lock or memory for it the answer is not kept
  try {
    std::lock_guard<std::mutex> lock(mutex);
    int& kept = known[std::make_tuple(kernel, threads, smem, dev)];            // 0: not asked yet
    if (kept == 0 && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem) == cudaSuccess && n > 0) kept = n;
    return kept > 0 ? kept : 1;
  } catch (const std::exception&) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem) == cudaSuccess && n > 0 ? n : 1;
  }
}
unsigned int* workspace_records(void* workspace, int64_t workspace_bytes, int64_t R, int64_t C) {
  const int64_t at = (metis_nvfp4_quantize_workspace_bytes(R, C) + 15) / 16 * 16;
  return workspace_bytes >= at + 16 + kMaxRecords * 12 ? reinterpret_cast<unsigned int*>(static_cast<char*>(workspace) + at) + 4 : nullptr;
}
static int sm_count() { return device_sm_count(); }

// *records: in: where the per-CTA records may go (or nullptr); out: nullptr if the running maximum was used instead
template <typename T>
static int32_t launch_rows(const T* x, int64_t rows, int64_t cols, int64_t ld, const float* mean, bool sr,
                           uint64_t seed, uint64_t offset, const uint64_t* ctr, uint32_t* codes, const WorkspaceView& ws,
                           cudaStream_t st, uint32_t sr16, unsigned int** records) {
  const int bpr = (int)(cols >> 4);
  auto kern = mean ? (sr ? quantize_rows_kernel<T, true, true> : quantize_rows_kernel<T, true, false>)
                   : (sr ? quantize_rows_kernel<T, false, true> : quantize_rows_kernel<T, false, false>);
  const int per_sm = resident_ctas(reinterpret_cast<const void*>(kern), kQuantThreads, 0);
  const RowsShape s = rows_shape(rows, bpr, (int64_t)sm_count() * per_sm, *records != nullptr);
  if (!s.records) {
    *records = nullptr;
    METIS_CUDA_OK(cudaMemsetAsync(ws.gmax, 0, 2 * sizeof(unsigned int), st));       // running maximum and error word
  }
  METIS_CUDA_OK(launch_overlapped(kLaunchStream, kern, dim3((unsigned)s.gx, (unsigned)s.gy), dim3((unsigned)s.bx, (unsigned)(kQuantThreads / s.bx)),
                                  0, st, x, (int)rows, bpr, ld, mean, PhiloxKeys(seed), offset, ctr, reinterpret_cast<uint2*>(codes), ws.amax, ws.gmax,
                                  *records, sr16));
  return METIS_OK;
}

template <typename T>
static int32_t launch_tile(const T* x, int64_t rows, int64_t cols, int64_t ld, const float* mean, bool sr,
                           uint64_t seed, uint64_t offset, const uint64_t* ctr, const TileOutputs& out, cudaStream_t st) {
  using TC = TileCfg<T>;
  CUtensorMap map;
  const CUtensorMapDataType dt = sizeof(T) == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  if (int32_t rc = make_map(&map, dt, sizeof(T), x, cols, rows, ld * (int64_t)sizeof(T), TC::kCols, TC::kRows, "x", 128))
    return rc;
  const int64_t col_tiles = ceil_div(cols, TC::kCols), tiles = col_tiles * ceil_div(rows, TC::kRows);
  if (tiles >= (int64_t)1 << 31) return fail(METIS_ERR_TOO_LARGE, "tensor of more than 2^31 tiles");
  const bool split_lines = (ld * (int64_t)sizeof(T)) % 128 != 0;
  int64_t grid = (int64_t)sm_count() * tile_ctas_per_sm(rows * ld * (int64_t)sizeof(T), split_lines, mean != nullptr, sizeof(T) == 4,
                                                          out.codes_r != nullptr, out.codes_t != nullptr);
  if (grid > tiles) grid = tiles;
  if (out.records && grid > kDualMaxCtas) grid = kDualMaxCtas;
  const uint32_t bpr = (uint32_t)(cols >> 4), bpc = (uint32_t)(rows >> 4), step_rows = (uint32_t)(grid / col_tiles), step_cols = (uint32_t)(grid % col_tiles);
  const TileWalk walk = {(uint32_t)tiles, (uint32_t)col_tiles, step_rows, step_cols, bpr, bpc,
                         step_rows * TC::kRows * bpr + step_cols * TC::kBlocksPerRow, TC::kRows * bpr - (uint32_t)col_tiles * TC::kBlocksPerRow,
                         step_cols * TC::kCols * bpc + step_rows * TC::kRowBlocks, TC::kRowBlocks - (uint32_t)col_tiles * TC::kCols * bpc};
  const PhiloxKeys keys(seed);
  const bool plain = !out.hadamard && !out.sr16;
  const bool with_rows = out.codes_r != nullptr, with_cols = out.codes_t != nullptr;
#define METIS_LAUNCH_TILE(MEAN, SR, ROWS, COLS, PLAIN)                                                      \
  do {                                                                                                      \
    auto kern = quantize_tile_kernel<T, MEAN, SR, ROWS, COLS, PLAIN>;                                       \
    METIS_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TC::kSmemBytes)); \
    METIS_CUDA_OK(launch_overlapped(kLaunchStream, kern, dim3((unsigned)grid), dim3(kQuantThreads), TC::kSmemBytes, st, map, walk, rows, cols, \
                                    mean, keys, offset, ctr, out));                                         \
  } while (0)
#define METIS_LAUNCH_TILE_MS(MEAN, SR)                                                                      \
  do {                                                                                                      \
    if (with_rows && with_cols) { if (plain) METIS_LAUNCH_TILE(MEAN, SR, true, true, true); else METIS_LAUNCH_TILE(MEAN, SR, true, true, false); } \
    else if (with_cols) { if (plain) METIS_LAUNCH_TILE(MEAN, SR, false, true, true); else METIS_LAUNCH_TILE(MEAN, SR, false, true, false); } \
    else if (plain || !SR) METIS_LAUNCH_TILE(MEAN, SR, true, false, true);                                  \
    else METIS_LAUNCH_TILE(MEAN, SR, true, false, !SR);                                                     \
  } while (0)
  if (mean) { if (sr) METIS_LAUNCH_TILE_MS(true, true); else METIS_LAUNCH_TILE_MS(true, false); }
  else      { if (sr) METIS_LAUNCH_TILE_MS(false, true); else METIS_LAUNCH_TILE_MS(false, false); }
#undef METIS_LAUNCH_TILE_MS
#undef METIS_LAUNCH_TILE
  return METIS_OK;
}

// Which kernel forms the row sums.  Four rows to a thread move the fewest bytes per instruction, but leave few CTAs where the
// tensor has few rows (16 per 128-row block), and where its last row block is not full the missing rows send that block
// down the edge path, a chain of loads per block; with 32 rows or fewer in it the tiled layout loses less there than the rows one
// by one lose to scattered words, and with many rows that chain is a small part.  Measured, dual quantizer with sums,
// four rows to a thread / threads of its own for each row (us): 16384 tokens x 128 columns 12.0 / 8.7, 65536 x 256 42.0 / 27.9,
// 65536 x 1024 106 / 90, 8192 x 1024 16.9 / 16.9, but 8192 x 1536 21.3 / 22.0, 16384 x 4096 89.9 / 94.7; last row block not
// full, tiled: 16384 x 2032 69.9 / 53.6, x 4144 113 / 105, 8192 x 7056 86.0 / 91.6, 10032 64.3 / 69.2; row-major: 9856 x 3744
// 62.7 / 56.8, 2176 x 8304 36.1 / 31.2, 256 x 14352 14.5 / 11.4, 4096 x 5056 34.8 / 36.7.
static bool rows_one_by_one(const FinalizeJob& J) {
  const int64_t last = J.R % 128;
  return J.R <= 1280 || (last != 0 && (J.sf_layout != METIS_SF_MMA || (last > 32 && J.R <= 8448)));
}

static FinalizeForm finalize_form(const FinalizeJobs& jobs, int njobs) {
  FinalizeForm form = kFinPlain;
  for (int j = 0; j < njobs; ++j) {
    const FinalizeJob& J = jobs.job[j];
    if (J.row_sums) return rows_one_by_one(J) ? kFinSumsByRow : kFinSums;          // one job at most wants them
    if (J.sf_cols % 4 != 0) form = kFinEdges;
  }
  return form;
}

static int32_t launch_finalize_jobs(FinalizeJobs jobs, int njobs, cudaStream_t st, uint64_t* offset_ctr) {
  const FinalizeForm form = finalize_form(jobs, njobs);
  int64_t blocks = 1;
  for (int j = 0; j < njobs; ++j) {
    FinalizeJob& J = jobs.job[j];
    const int64_t groups = J.sf_layout == METIS_SF_MMA ? sf_tiles_per_row(J.sf_cols * 16) : ceil_div(J.sf_cols, 4);
    const bool by_row = form == kFinSumsByRow && J.row_sums;
    J.log_tx = 2;                                             // a warp holds at most 8 rows' lanes of 4 tiles
    while (J.log_tx < (by_row ? 7 : 6) && (1 << J.log_tx) < groups) ++J.log_tx;
    // Rows one by one: fewer threads to a row where that leaves fewer of them idle in its last round and the rows still give
    // every SM 256 of them.  2176 tokens (34 groups of blocks, 16 threads for 64) x 5056 columns 25.8 -> 21.2 us (tiled), 9856
    // (154, 32 for 128) x 3744 63.0 -> 56.8 (row-major).
    if (by_row) {
      auto lanes = [&](int log_tx) { return (((groups - 1) >> log_tx) + 1) << log_tx; };
      for (int l = J.log_tx - 1; l >= 3 && (J.R << l) >= (int64_t)sm_count() * 256; --l) if (lanes(l) < lanes(J.log_tx)) J.log_tx = l;
    }
    const int64_t segments = J.row_sums ? 1 : ceil_div(groups, (int64_t)1 << J.log_tx);
    const int64_t need = by_row ? ceil_div(ceil_div(J.R, 128) * 128, kFinThreads >> J.log_tx)
                                : ceil_div(ceil_div(J.R, 128) * 16 * segments, 64 >> J.log_tx);
    if (need > blocks) blocks = need;
  }
  if (njobs == 1) jobs.job[1] = jobs.job[0];
  const bool sums = form == kFinSums || form == kFinSumsByRow;
  auto kern = form == kFinPlain ? finalize_scales_kernel<kFinPlain> : form == kFinEdges ? finalize_scales_kernel<kFinEdges>
            : form == kFinSums ? finalize_scales_sums_kernel : finalize_scales_kernel<kFinSumsByRow>;
  const int64_t cap = (int64_t)sm_count() * (sums ? 10 : 8) / njobs;     // resident at once: 5 (sums) and 8 per SM
  if (blocks > cap) blocks = ceil_div(blocks, ceil_div(blocks, cap));    // the fewest CTAs that need no more rounds than `cap` would
  METIS_CUDA_OK(launch_overlapped(kLaunchShort, kern, dim3((unsigned)blocks, (unsigned)njobs), dim3(kFinThreads), 0, st,
                                  jobs.job[0], jobs.job[1], offset_ctr));
  return METIS_OK;
}

int32_t launch_finalize(const WorkspaceView& ws, int64_t R, int64_t C, int32_t sf_layout, uint8_t* scales, float* unit,
                        cudaStream_t st, uint64_t* offset_ctr, const unsigned int* records, int32_t which) {
  FinalizeJobs jobs = {};
  jobs.job[0] = {ws.amax, ws.gmax, ws.gmax + 1, R, C / 16, sf_layout, scales, unit, 0, nullptr, nullptr, records, which};
  return launch_finalize_jobs(jobs, 1, st, offset_ctr);
}

int32_t check_quant_outputs(int64_t R, int64_t C, int32_t sf_layout, const void* codes,
                            const void* scales, const void* unit, const void* workspace,
                            int64_t workspace_bytes) {
  if (R <= 0 || C <= 0) return fail(METIS_ERR_BAD_SHAPE, "empty tensor [%lld, %lld]", (long long)R, (long long)C);
  if (C % 16 != 0)
    return fail(METIS_ERR_BAD_SHAPE, "NVFP4 block shape (1, 16) does not divide tensor shape (%lld, %lld)",
                (long long)R, (long long)C);
  if (sf_layout != METIS_SF_ROWMAJOR && sf_layout != METIS_SF_MMA)
    return fail(METIS_ERR_BAD_ARGUMENT, "unknown sf_layout %d", sf_layout);
  if (!codes || !scales || !unit || !workspace) return fail(METIS_ERR_BAD_ARGUMENT, "null output pointer");
  if (!aligned16(codes) || !aligned16(scales) || !aligned16(workspace))
    return fail(METIS_ERR_BAD_ALIGNMENT, "codes, scales and workspace must be 16-byte aligned");
  if (workspace_bytes < metis_nvfp4_quantize_workspace_bytes(R, C))
    return fail(METIS_ERR_WORKSPACE, "workspace of %lld bytes, need %lld", (long long)workspace_bytes,
                (long long)metis_nvfp4_quantize_workspace_bytes(R, C));
  return METIS_OK;
}

}  // namespace metis

using namespace metis;

extern "C" int64_t metis_nvfp4_sf_bytes(int64_t R, int64_t C, int32_t sf_layout) {
  if (R <= 0 || C <= 0) return 0;
  if (sf_layout == METIS_SF_MMA) return ceil_div(R, 128) * sf_tiles_per_row(C) * 512;
  return R * ceil_div(C, 16);
}

extern "C" int64_t metis_nvfp4_quantize_workspace_bytes(int64_t R, int64_t C) {
  if (R <= 0 || C <= 0) return kHeaderBytes;
  return kHeaderBytes + R * ceil_div(C, 16) * (int64_t)sizeof(float);
}

extern "C" int32_t metis_nvfp4_quantize(const void* x, int32_t x_dtype, int64_t rows, int64_t cols,
                                        int64_t ld, const float* col_mean, uint32_t flags,
                                        uint64_t seed, uint64_t offset, int32_t sf_layout,
                                        uint8_t* codes, uint8_t* scales, float* unit, void* workspace,
                                        int64_t workspace_bytes, void* stream) {
  const bool transpose = flags & METIS_Q_TRANSPOSE;
  const bool sr = flags & METIS_Q_STOCHASTIC;
  // graph-safe random stream: `offset` carries the address of a device counter instead of a value
  uint64_t* ctr = (sr && (flags & METIS_Q_OFFSET_ON_DEVICE)) ? reinterpret_cast<uint64_t*>(static_cast<uintptr_t>(offset)) : nullptr;
  if (ctr) offset = 0;
  if ((flags & METIS_Q_OFFSET_ON_DEVICE) && (!sr || !ctr || (reinterpret_cast<uintptr_t>(ctr) & 7u)))
    return fail(METIS_ERR_BAD_ARGUMENT, "METIS_Q_OFFSET_ON_DEVICE needs METIS_Q_STOCHASTIC and an 8-byte aligned device address in offset");
  if (flags & ~(METIS_Q_TRANSPOSE | METIS_Q_STOCHASTIC | METIS_Q_OFFSET_ON_DEVICE | METIS_Q_HADAMARD | METIS_Q_SIGN_MASK | METIS_Q_SR16)) return fail(METIS_ERR_BAD_ARGUMENT, "unknown flags 0x%x", flags);
  if ((flags & METIS_Q_SR16) && !sr) return fail(METIS_ERR_BAD_ARGUMENT, "METIS_Q_SR16 without METIS_Q_STOCHASTIC");
  const uint32_t sr16 = (flags & METIS_Q_SR16) ? 1u : 0u;
  if ((flags & METIS_Q_HADAMARD) && !transpose) return fail(METIS_ERR_UNSUPPORTED, "METIS_Q_HADAMARD rotates the blocks of the transposed quantization: it needs METIS_Q_TRANSPOSE");
  if ((flags & METIS_Q_SIGN_MASK) && !(flags & METIS_Q_HADAMARD)) return fail(METIS_ERR_BAD_ARGUMENT, "sign bits without METIS_Q_HADAMARD");
  const uint32_t rht = (flags & METIS_Q_HADAMARD) ? ((1u << 16) | (flags >> 16)) : 0u;
  if (!x) return fail(METIS_ERR_BAD_ARGUMENT, "x is null");
  if (x_dtype != METIS_DTYPE_BF16 && x_dtype != METIS_DTYPE_F32) return fail(METIS_ERR_BAD_ARGUMENT, "unknown x_dtype %d", x_dtype);
  if (rows <= 0 || cols <= 0) return fail(METIS_ERR_BAD_SHAPE, "empty tensor [%lld, %lld]", (long long)rows, (long long)cols);
  if (ld < cols) return fail(METIS_ERR_BAD_ARGUMENT, "ld %lld < cols %lld", (long long)ld, (long long)cols);
  const int64_t R = transpose ? cols : rows, C = transpose ? rows : cols;
  if (int32_t rc = check_quant_outputs(R, C, sf_layout, codes, scales, unit, workspace, workspace_bytes)) return rc;
  const int64_t esz = x_dtype == METIS_DTYPE_BF16 ? 2 : 4;
  // vector loads: 8 elements per thread row-major, 16 bytes per thread transposed
  const int64_t need = transpose ? 16 / esz : 8;
  if (cols % need != 0 || ld % need != 0 || !aligned16(x))
    return fail(METIS_ERR_BAD_ALIGNMENT, "x must be 16-byte aligned with cols and ld multiples of %lld", (long long)need);
  if (col_mean && !aligned16(col_mean)) return fail(METIS_ERR_BAD_ALIGNMENT, "col_mean must be 16-byte aligned");
  if (rows >= ((int64_t)1 << 31) || cols >= ((int64_t)1 << 31)) return fail(METIS_ERR_TOO_LARGE, "tensor too large");
  if (rows * cols >= kMaxElements) return fail(METIS_ERR_TOO_LARGE, "tensor of 2^36 elements or more");

  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // With METIS_QUANTIZE_EXTRA_WORKSPACE bytes more than it needs the workspace also holds a record per CTA of the first
  // pass, as in the dual quantizer; without them the running maximum and the error word are zeroed in front of it, and
  // that memset node costs 3-4 us (16 x 14336: 8.2 us with it, 4.9 without; 1120 x 3584: 12.4, 8.1).
  unsigned int* records = workspace_records(workspace, workspace_bytes, R, C);
  // One cluster for the whole tensor; with records, only where two launches over many SMs are not faster.
  int64_t tiles = 0, padded_words = 0;
  if (!transpose && !sr && aligned16(scales) && small_path(R, C, sf_layout, &tiles, &padded_words) &&
      (!records || R * (C / 16) <= cluster_blocks(C, sf_layout, esz))) {
    return x_dtype == METIS_DTYPE_BF16
        ? launch_small(static_cast<const __nv_bfloat16*>(x), rows, cols, ld, col_mean, codes, sf_layout, tiles, padded_words, scales, unit, st)
        : launch_small(static_cast<const float*>(x), rows, cols, ld, col_mean, codes, sf_layout, tiles, padded_words, scales, unit, st);
  }
  const WorkspaceView ws = view_workspace(workspace);
  // Large row-major tensors take the tile kernel too (row phase only): its TMA ring keeps two tiles in
  // flight per CTA, where the register-fed kernel waits on its loads.  Same arithmetic, same bytes.
  const bool rows_by_tiles = !transpose && rows * cols >= kTileRowsMinElements && (ld * esz) % 16 == 0;
  int32_t rc;
  if (transpose || rows_by_tiles) {
    if (!records) METIS_CUDA_OK(cudaMemsetAsync(ws.gmax, 0, 2 * sizeof(unsigned int), st));     // running maximum and error word
    TileOutputs out = {};
    if (transpose) { out.codes_t = codes; out.amax_t = ws.amax; out.gmax_t = ws.gmax; out.hadamard = rht; }
    else           { out.codes_r = codes; out.amax_r = ws.amax; out.gmax_r = ws.gmax; }
    out.error = ws.gmax + 1;
    out.records = records;
    out.sr16 = sr16;
    rc = x_dtype == METIS_DTYPE_BF16
        ? launch_tile(static_cast<const __nv_bfloat16*>(x), rows, cols, ld, col_mean, sr, seed, offset, ctr, out, st)
        : launch_tile(static_cast<const float*>(x), rows, cols, ld, col_mean, sr, seed, offset, ctr, out, st);
  } else {
    rc = x_dtype == METIS_DTYPE_BF16
        ? launch_rows(static_cast<const __nv_bfloat16*>(x), rows, cols, ld, col_mean, sr, seed, offset, ctr,
                      reinterpret_cast<uint32_t*>(codes), ws, st, sr16, &records)
        : launch_rows(static_cast<const float*>(x), rows, cols, ld, col_mean, sr, seed, offset, ctr,
                      reinterpret_cast<uint32_t*>(codes), ws, st, sr16, &records);
  }
  if (rc) return rc;
  METIS_CUDA_OK(cudaGetLastError());
  return launch_finalize(ws, R, C, sf_layout, scales, unit, st, ctr, records, transpose ? 1 : 0);
}

// Scale pass of the dual quantizer's outputs (either or both) from the block maxima in its workspace.
static int32_t finish_dual(int64_t rows, int64_t cols, int32_t sf_layout, uint8_t* scales, float* unit, const uint8_t* codes_t,
                           uint8_t* scales_t, float* unit_t, float* token_sums_t, void* workspace, bool rowmajor,
                           bool transposed, cudaStream_t st, uint64_t* ctr) {
  const unsigned int* records = static_cast<const unsigned int*>(workspace) + 64;
  float* amax_r = reinterpret_cast<float*>(static_cast<char*>(workspace) + kDualHeaderBytes);
  float* amax_t = amax_r + rows * (cols / 16);
  FinalizeJobs jobs = {};
  int n = 0;
  // The job with sums first: its CTAs run longer, and the others fill the SMs that they leave (16384 x 4096, stochastic, both with
  // sums 97.1 -> 94.6 us; 16384 x 2032 50.5 -> 48.8; row-major 4096 x 5056 36.6 -> 33.9).
  if (transposed)
    jobs.job[n++] = {amax_t, nullptr, nullptr, cols, rows / 16, sf_layout, scales_t, unit_t, 0,
                     token_sums_t ? reinterpret_cast<const uint2*>(codes_t) : nullptr, token_sums_t, records, 1};
  if (rowmajor) jobs.job[n++] = {amax_r, nullptr, nullptr, rows, cols / 16, sf_layout, scales, unit, 0, nullptr, nullptr, records, 0};
  if (n == 0) return METIS_OK;
  return launch_finalize_jobs(jobs, n, st, ctr);      // job 0 of the launch bumps the Philox offset counter, if there is one
}

extern "C" int64_t metis_nvfp4_quantize_dual_workspace_bytes(int64_t rows, int64_t cols) {
  if (rows <= 0 || cols <= 0) return kDualHeaderBytes;
  return kDualHeaderBytes + 2 * rows * ceil_div(cols, 16) * (int64_t)sizeof(float);
}

extern "C" int32_t metis_nvfp4_quantize_dual(const void* x, int32_t x_dtype, int64_t rows, int64_t cols, int64_t ld,
                                             const float* col_mean, uint32_t flags, uint64_t seed, uint64_t offset,
                                             int32_t sf_layout, uint8_t* codes, uint8_t* scales, float* unit,
                                             uint8_t* codes_t, uint8_t* scales_t, float* unit_t, float* token_sums_t,
                                             void* workspace, int64_t workspace_bytes, void* stream) {
  const bool sr = flags & METIS_Q_STOCHASTIC;
  uint64_t* ctr = (sr && (flags & METIS_Q_OFFSET_ON_DEVICE)) ? reinterpret_cast<uint64_t*>(static_cast<uintptr_t>(offset)) : nullptr;
  if (ctr) offset = 0;
  if ((flags & METIS_Q_OFFSET_ON_DEVICE) && (!sr || !ctr || (reinterpret_cast<uintptr_t>(ctr) & 7u)))
    return fail(METIS_ERR_BAD_ARGUMENT, "METIS_Q_OFFSET_ON_DEVICE needs METIS_Q_STOCHASTIC and an 8-byte aligned device address in offset");
  if (flags & ~(METIS_Q_STOCHASTIC | METIS_Q_OFFSET_ON_DEVICE | METIS_Q_HADAMARD | METIS_Q_SIGN_MASK | METIS_Q_DEFER_ROWMAJOR | METIS_Q_DEFER_TRANSPOSED | METIS_Q_SR16)) return fail(METIS_ERR_BAD_ARGUMENT, "unknown flags 0x%x (the dual quantizer always writes both orientations)", flags);
  if ((flags & METIS_Q_SR16) && !sr) return fail(METIS_ERR_BAD_ARGUMENT, "METIS_Q_SR16 without METIS_Q_STOCHASTIC");
  if ((flags & METIS_Q_DEFER_ROWMAJOR) && (flags & METIS_Q_DEFER_TRANSPOSED)) return fail(METIS_ERR_BAD_ARGUMENT, "only one of the two scale passes can be deferred");
  if ((flags & METIS_Q_SIGN_MASK) && !(flags & METIS_Q_HADAMARD)) return fail(METIS_ERR_BAD_ARGUMENT, "sign bits without METIS_Q_HADAMARD");
  const uint32_t rht = (flags & METIS_Q_HADAMARD) ? ((1u << 16) | (flags >> 16)) : 0u;      // the transposed output only
  if (token_sums_t && rht) return fail(METIS_ERR_BAD_ARGUMENT, "token_sums_t is not available with METIS_Q_HADAMARD (the rotated blocks need weighted sums)");
  if (token_sums_t && rows % 64 != 0) return fail(METIS_ERR_BAD_SHAPE, "token_sums_t needs rows to be a multiple of 64");
  if (!x) return fail(METIS_ERR_BAD_ARGUMENT, "x is null");
  if (x_dtype != METIS_DTYPE_BF16 && x_dtype != METIS_DTYPE_F32) return fail(METIS_ERR_BAD_ARGUMENT, "unknown x_dtype %d", x_dtype);
  if (rows <= 0 || cols <= 0) return fail(METIS_ERR_BAD_SHAPE, "empty tensor [%lld, %lld]", (long long)rows, (long long)cols);
  if (rows % 16 != 0 || cols % 16 != 0)
    return fail(METIS_ERR_BAD_SHAPE, "NVFP4 block shape (1, 16) does not divide both dimensions of tensor shape (%lld, %lld)", (long long)rows, (long long)cols);
  if (ld < cols) return fail(METIS_ERR_BAD_ARGUMENT, "ld %lld < cols %lld", (long long)ld, (long long)cols);
  if (sf_layout != METIS_SF_ROWMAJOR && sf_layout != METIS_SF_MMA) return fail(METIS_ERR_BAD_ARGUMENT, "unknown sf_layout %d", sf_layout);
  if (!codes || !scales || !unit || !codes_t || !scales_t || !unit_t || !workspace) return fail(METIS_ERR_BAD_ARGUMENT, "null output pointer");
  const int64_t esz = x_dtype == METIS_DTYPE_BF16 ? 2 : 4;
  if (ld % (16 / esz) != 0 || !aligned16(x) || !aligned16(codes) || !aligned16(scales) || !aligned16(codes_t) || !aligned16(scales_t) || !aligned16(workspace))
    return fail(METIS_ERR_BAD_ALIGNMENT, "x, codes, scales and workspace must be 16-byte aligned, rows of x too");
  if (col_mean && !aligned16(col_mean)) return fail(METIS_ERR_BAD_ALIGNMENT, "col_mean must be 16-byte aligned");
  if (workspace_bytes < metis_nvfp4_quantize_dual_workspace_bytes(rows, cols))
    return fail(METIS_ERR_WORKSPACE, "workspace of %lld bytes, need %lld", (long long)workspace_bytes,
                (long long)metis_nvfp4_quantize_dual_workspace_bytes(rows, cols));
  if (rows >= ((int64_t)1 << 31) || cols >= ((int64_t)1 << 31)) return fail(METIS_ERR_TOO_LARGE, "tensor too large");
  if (rows * cols >= kMaxElements) return fail(METIS_ERR_TOO_LARGE, "tensor of 2^36 elements or more");

  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // every CTA of the first pass leaves its maxima and its error word in a record of its own: nothing to zero first
  unsigned int* records = static_cast<unsigned int*>(workspace) + 64;
  float* amax_r = reinterpret_cast<float*>(static_cast<char*>(workspace) + kDualHeaderBytes);
  float* amax_t = amax_r + rows * (cols / 16);
  const TileOutputs out = {codes_t, amax_t, nullptr, codes, amax_r, nullptr, nullptr, records, rht, (flags & METIS_Q_SR16) ? 1u : 0u};
  const int32_t rc = x_dtype == METIS_DTYPE_BF16
      ? launch_tile(static_cast<const __nv_bfloat16*>(x), rows, cols, ld, col_mean, sr, seed, offset, ctr, out, st)
      : launch_tile(static_cast<const float*>(x), rows, cols, ld, col_mean, sr, seed, offset, ctr, out, st);
  if (rc) return rc;
  METIS_CUDA_OK(cudaGetLastError());
  return finish_dual(rows, cols, sf_layout, scales, unit, codes_t, scales_t, unit_t, token_sums_t, workspace,
                     !(flags & METIS_Q_DEFER_ROWMAJOR), !(flags & METIS_Q_DEFER_TRANSPOSED), st, ctr);
}

extern "C" int32_t metis_nvfp4_quantize_dual_finish(int64_t rows, int64_t cols, uint32_t deferred, int32_t sf_layout,
                                                    uint8_t* scales, float* unit, const uint8_t* codes_t, uint8_t* scales_t,
                                                    float* unit_t, float* token_sums_t, void* workspace,
                                                    int64_t workspace_bytes, void* stream) {
  const bool rowmajor = deferred == METIS_Q_DEFER_ROWMAJOR, transposed = deferred == METIS_Q_DEFER_TRANSPOSED;
  if (!rowmajor && !transposed) return fail(METIS_ERR_BAD_ARGUMENT, "deferred must be METIS_Q_DEFER_ROWMAJOR or METIS_Q_DEFER_TRANSPOSED");
  if (rows <= 0 || cols <= 0 || rows % 16 != 0 || cols % 16 != 0) return fail(METIS_ERR_BAD_SHAPE, "bad shape [%lld, %lld]", (long long)rows, (long long)cols);
  if (sf_layout != METIS_SF_ROWMAJOR && sf_layout != METIS_SF_MMA) return fail(METIS_ERR_BAD_ARGUMENT, "unknown sf_layout %d", sf_layout);
  if (!workspace || !aligned16(workspace) || workspace_bytes < metis_nvfp4_quantize_dual_workspace_bytes(rows, cols))
    return fail(METIS_ERR_WORKSPACE, "the workspace of the quantizing call is needed");
  if (rowmajor && (!scales || !unit || !aligned16(scales))) return fail(METIS_ERR_BAD_ARGUMENT, "scales and unit of the row-major output");
  if (transposed && (!scales_t || !unit_t || !aligned16(scales_t) || (token_sums_t && !codes_t)))
    return fail(METIS_ERR_BAD_ARGUMENT, "scales_t and unit_t of the transposed output (and codes_t for token_sums_t)");
  if (token_sums_t && rows % 64 != 0) return fail(METIS_ERR_BAD_SHAPE, "token_sums_t needs rows to be a multiple of 64");
  return finish_dual(rows, cols, sf_layout, scales, unit, codes_t, scales_t, unit_t, token_sums_t, workspace,
                     rowmajor, transposed, reinterpret_cast<cudaStream_t>(stream), nullptr);
}

extern "C" int64_t metis_col_mean_workspace_bytes(int64_t rows, int64_t cols) {
  if (rows <= 0 || cols <= 0) return 0;
  return col_mean_splits(rows) * cols * (int64_t)sizeof(float);
}

extern "C" int32_t metis_col_mean(const void* x, int32_t x_dtype, int64_t rows, int64_t cols, int64_t ld,
                                  float* mean, void* workspace, int64_t workspace_bytes, void* stream) {
  if (!x || !mean || !workspace) return fail(METIS_ERR_BAD_ARGUMENT, "null pointer");
  if (x_dtype != METIS_DTYPE_BF16 && x_dtype != METIS_DTYPE_F32) return fail(METIS_ERR_BAD_ARGUMENT, "unknown x_dtype %d", x_dtype);
  if (rows <= 0 || cols <= 0) return fail(METIS_ERR_BAD_SHAPE, "empty tensor");
  if (cols % 8 != 0 || ld % 8 != 0 || ld < cols || !aligned16(x))
    return fail(METIS_ERR_BAD_ALIGNMENT, "x must be 16-byte aligned with cols and ld multiples of 8");
  if (workspace_bytes < metis_col_mean_workspace_bytes(rows, cols))
    return fail(METIS_ERR_WORKSPACE, "workspace too small");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int64_t splits = col_mean_splits(rows);
  const int64_t rows_per_split = ceil_div(rows, splits);
  const dim3 g((unsigned)ceil_div(cols, 256), (unsigned)splits);
  // up to 128 rows there is one split: stage 1 writes the mean itself (0 + sum, then the same division)
  const bool single = splits == 1;
  float* partial = single ? mean : static_cast<float*>(workspace);
  const int64_t mean_of_rows = single ? rows : 0;
  if (x_dtype == METIS_DTYPE_BF16)
    METIS_CUDA_OK(launch_overlapped(kLaunchStream, col_partial_sum_kernel<__nv_bfloat16>, g, dim3(kMeanThreads), 0, st,
                                    static_cast<const __nv_bfloat16*>(x), rows, cols, ld, rows_per_split, partial, mean_of_rows));
  else
    METIS_CUDA_OK(launch_overlapped(kLaunchStream, col_partial_sum_kernel<float>, g, dim3(kMeanThreads), 0, st,
                                    static_cast<const float*>(x), rows, cols, ld, rows_per_split, partial, mean_of_rows));
  if (!single)
    METIS_CUDA_OK(launch_overlapped(kLaunchShort, col_mean_finish_kernel, dim3((unsigned)ceil_div(cols, 256)), dim3(256), 0, st,
                                    partial, splits, rows, cols, mean));
  return METIS_OK;
}

// ---- quantizer entry point that brings its own scratch -----------------------------------------------
//
// metis_nvfp4_quantize needs a caller-provided workspace for the per-block maxima.  Some callers
// have no way to provide one: a serving loop whose device memory was carved up once at start-up
// and must not grow, a host binding (cgo, JNI) that holds raw device pointers but no allocator, a
// latency-critical section in which cudaMalloc's implicit device synchronisation is not acceptable.
// For them the scratch lives in this translation unit as a fixed-size device array; the price is
// that every GPU that loads the library keeps these bytes until the process exits, and that the
// tensor size is capped.
namespace metis {

constexpr int64_t kStaticMaxElements = METIS_STATIC_MAX_ELEMENTS;                        // 16 Mi elements
constexpr int64_t kStaticScratchBytes = kWorkspaceHeaderBytes + (kStaticMaxElements / 16) * 4;  // 4 MiB + 256 B

// In device code this name is the array.  In host code it is only a handle for the runtime's symbol
// table, NOT a device address: the address is looked up below with cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

constexpr int kMaxDevices = 64;
static void* g_static_scratch_addr[kMaxDevices] = {};
static std::mutex g_static_scratch_mutex;

// Device address of the array on the CURRENT device, resolved once per device.
static int32_t static_scratch_address(void** out) {
  int dev = -1;
  METIS_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail(METIS_ERR_UNSUPPORTED, "device index %d is outside [0, %d)", dev, kMaxDevices);
  std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
  if (g_static_scratch_addr[dev] == nullptr) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess || p == nullptr)
      return fail(METIS_ERR_CUDA, "cudaGetSymbolAddress(static scratch) on device %d: %s", dev, cudaGetErrorString(e));
    g_static_scratch_addr[dev] = p;
  }
  *out = g_static_scratch_addr[dev];
  return METIS_OK;
}

}  // namespace metis

extern "C" int32_t metis_nvfp4_quantize_static(const void* x, int32_t x_dtype, int64_t rows, int64_t cols,
                                               int64_t ld, int32_t sf_layout, uint8_t* codes,
                                               uint8_t* scales, float* unit, void* stream) {
  if (!x) return fail(METIS_ERR_BAD_ARGUMENT, "x is null");
  if (x_dtype != METIS_DTYPE_BF16 && x_dtype != METIS_DTYPE_F32) return fail(METIS_ERR_BAD_ARGUMENT, "unknown x_dtype %d", x_dtype);
  if (rows <= 0 || cols <= 0) return fail(METIS_ERR_BAD_SHAPE, "empty tensor [%lld, %lld]", (long long)rows, (long long)cols);
  if (cols % 16 != 0)
    return fail(METIS_ERR_BAD_SHAPE, "NVFP4 block shape (1, 16) does not divide tensor shape (%lld, %lld)", (long long)rows, (long long)cols);
  if (rows > kStaticMaxElements / cols)
    return fail(METIS_ERR_TOO_LARGE, "%lld x %lld elements exceed the built-in scratch (METIS_STATIC_MAX_ELEMENTS = %lld); "
                "use metis_nvfp4_quantize with a caller workspace", (long long)rows, (long long)cols, (long long)kStaticMaxElements);
  if (ld < cols) return fail(METIS_ERR_BAD_ARGUMENT, "ld %lld < cols %lld", (long long)ld, (long long)cols);
  if (sf_layout != METIS_SF_ROWMAJOR && sf_layout != METIS_SF_MMA) return fail(METIS_ERR_BAD_ARGUMENT, "unknown sf_layout %d", sf_layout);
  if (!codes || !scales || !unit) return fail(METIS_ERR_BAD_ARGUMENT, "null output pointer");
  if (ld % 8 != 0 || !aligned16(x) || !aligned16(codes) || !aligned16(scales))
    return fail(METIS_ERR_BAD_ALIGNMENT, "x, codes and scales must be 16-byte aligned and ld a multiple of 8");

  void* scratch = nullptr;
  if (int32_t rc = static_scratch_address(&scratch)) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const WorkspaceView ws = view_workspace(scratch);
  // The array keeps whatever the previous call left.  Only the running maximum and the error word
  // have to start at zero; every block maximum this call reads back is written by this call first.
  unsigned int* records = nullptr;                      // the built-in scratch has no room for them
  const int32_t rc = x_dtype == METIS_DTYPE_BF16
      ? launch_rows(static_cast<const __nv_bfloat16*>(x), rows, cols, ld, nullptr, false, 0, 0, nullptr, reinterpret_cast<uint32_t*>(codes), ws, st, 0u, &records)
      : launch_rows(static_cast<const float*>(x), rows, cols, ld, nullptr, false, 0, 0, nullptr, reinterpret_cast<uint32_t*>(codes), ws, st, 0u, &records);
  if (rc) return rc;
  METIS_CUDA_OK(cudaGetLastError());
  return launch_finalize(ws, rows, cols, sf_layout, scales, unit, st);
}

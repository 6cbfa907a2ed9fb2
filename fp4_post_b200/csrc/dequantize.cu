// NVFP4 -> dense conversion and the quantized matrix x vector product.
#include "common.cuh"

#include <cuda_fp16.h>

namespace metis {

__device__ __forceinline__ float scale_at(const uint8_t* scales, int32_t sf_layout, int64_t r,
                                          int64_t k, int64_t sf_cols, int64_t tiles) {
  const int64_t off = (sf_layout == METIS_SF_MMA) ? sf_mma_offset(r, k, tiles) : r * sf_cols + k;
  return e4m3_to_float(__ldg(scales + off));
}

// The unit the values are expressed in: *u0, or (*u0 * *u1) / (*d0 * *d1) (a ratio of two products' units, formed here
// instead of by three one-element kernels in front of this one).
struct UnitPtrs {
  const float* u0;  const float* u1;  const float* d0;  const float* d1;
};

// One thread per 8 elements (4 code bytes).  kRatio: the unit is the ratio of four.  A kernel of its own: a small call feels the
// test (622 x 944 to bf16 1.72 us with it, 1.68 without; 4261 x 256 2.48 and 2.40).
template <typename TO, bool kRatio>
__global__ void __launch_bounds__(256)
dequantize_kernel(const uint32_t* __restrict__ codes, const uint8_t* __restrict__ scales,
                  const UnitPtrs units, int32_t sf_layout, int64_t R, int64_t C,
                  const float* __restrict__ add_row_vec, TO* __restrict__ out, int64_t ld) {
  grid_dependency_wait();
  float unit = __ldg(units.u0);
  if constexpr (kRatio) unit = __fdiv_rn(__fmul_rn(unit, __ldg(units.u1)), __fmul_rn(__ldg(units.d0), __ldg(units.d1)));
  const int64_t chunks_per_row = C >> 3;
  const int64_t total = R * chunks_per_row;
  const bool small = total < ((int64_t)1 << 31);
  const int64_t sf_cols = C >> 4;
  const int64_t tiles = sf_tiles_per_row(C);
  for (int64_t c = (int64_t)blockIdx.x * 256 + threadIdx.x; c < total; c += (int64_t)gridDim.x * 256) {
    // 32-bit index arithmetic where it fits (a 64-bit division is a subroutine of ~100 instructions)
    const int64_t r = small ? (int64_t)((uint32_t)c / (uint32_t)chunks_per_row) : c / chunks_per_row;
    const int64_t ch = c - r * chunks_per_row;
    const uint32_t w = __ldg(codes + c);
    // value = e2m1 * (e4m3 * unit): the same two roundings as quant.py:23-35
    const float d = __fmul_rn(scale_at(scales, sf_layout, r, ch >> 1, sf_cols, tiles), unit);
    float y[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t nib = (w >> (4 * i)) & 15u;
      float val = __fmul_rn(e2m1_value(nib & 7u), d);
      if (nib & 8u) val = -val;
      y[i] = val;
    }
    if (add_row_vec) {
#pragma unroll
      for (int i = 0; i < 8; ++i) y[i] = __fadd_rn(__ldg(add_row_vec + ch * 8 + i), y[i]);
    }
    TO* dst = out + r * ld + ch * 8;
    if constexpr (sizeof(TO) == 2) {
      __nv_bfloat162 o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) o[i] = __floats2bfloat162_rn(y[2 * i], y[2 * i + 1]);
      *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<uint4*>(o);
    } else {
      reinterpret_cast<float4*>(dst)[0] = make_float4(y[0], y[1], y[2], y[3]);
      reinterpret_cast<float4*>(dst)[1] = make_float4(y[4], y[5], y[6], y[7]);
    }
  }
}

// out[r] = sum_c v[c] * value(Q[r][c]).  One warp per row; per step a lane takes one block (16
// elements: one 64-bit load of codes, one scale byte), so a warp reads 512 consecutive elements and
// the matching stretch of v with 128-bit loads.  Twice the e2m1 magnitude comes from a nibble table
// held in one 32-bit constant; a block's partial sum is formed in integers (v == NULL) or with one
// multiply-add per element, then scaled once.
__device__ __forceinline__ int twice_e2m1(uint32_t nib) {
  const int mag = (int)((0xC8643210u >> ((nib & 7u) * 4u)) & 15u);     // {0,1,2,3,4,6,8,12}
  return (nib & 8u) ? -mag : mag;
}

template <bool kHasV>
__global__ void __launch_bounds__(256)
gemv_kernel(const uint2* __restrict__ codes, const uint8_t* __restrict__ scales,
            const float* __restrict__ unit_ptr, int32_t sf_layout, int64_t R, int64_t C,
            const float* __restrict__ v, float* __restrict__ out) {
  grid_dependency_wait();
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= R) return;
  const int64_t sf_cols = C >> 4;               // blocks per row
  const int64_t tiles = sf_tiles_per_row(C);
  const uint2* row_codes = codes + row * sf_cols;
  float acc = 0.0f;
  if (!kHasV && sf_layout == METIS_SF_MMA && (sf_cols & 3) == 0) {
    // row sums: four blocks per lane and trip (two 16-byte loads of codes, the four scale bytes
    // are one aligned word of the tile layout)
#pragma unroll 2
    for (int64_t g = lane; g < (sf_cols >> 2); g += 32) {
      const uint4 a = __ldg(reinterpret_cast<const uint4*>(row_codes + 4 * g));
      const uint4 b = __ldg(reinterpret_cast<const uint4*>(row_codes + 4 * g) + 1);
      const uint32_t s4 = __ldg(reinterpret_cast<const uint32_t*>(scales + sf_mma_offset(row, 4 * g, tiles)));
      acc = fmaf((float)block_code_sum(make_uint2(a.x, a.y)), e4m3_to_float(s4 & 0xFFu), acc);
      acc = fmaf((float)block_code_sum(make_uint2(a.z, a.w)), e4m3_to_float((s4 >> 8) & 0xFFu), acc);
      acc = fmaf((float)block_code_sum(make_uint2(b.x, b.y)), e4m3_to_float((s4 >> 16) & 0xFFu), acc);
      acc = fmaf((float)block_code_sum(make_uint2(b.z, b.w)), e4m3_to_float(s4 >> 24), acc);
    }
  } else
#pragma unroll 4
  for (int64_t k = lane; k < sf_cols; k += 32) {
    const uint2 w2 = __ldg(row_codes + k);
    const int64_t off = (sf_layout == METIS_SF_MMA) ? sf_mma_offset(row, k, tiles) : row * sf_cols + k;
    const float sc = e4m3_to_float(__ldg(scales + off));
    const uint32_t w[2] = {w2.x, w2.y};
    float part;
    if (kHasV) {
      part = 0.0f;
      const float4* v4 = reinterpret_cast<const float4*>(v + k * 16);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 f = __ldg(v4 + j);
        const uint32_t n4 = w[j >> 1] >> (16 * (j & 1));
        part = fmaf((float)twice_e2m1(n4), f.x, part);
        part = fmaf((float)twice_e2m1(n4 >> 4), f.y, part);
        part = fmaf((float)twice_e2m1(n4 >> 8), f.z, part);
        part = fmaf((float)twice_e2m1(n4 >> 12), f.w, part);
      }
    } else {
      part = (float)block_code_sum(w2);
    }
    acc = fmaf(part, sc, acc);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) out[row] = acc * (0.5f * __ldg(unit_ptr));
}

__device__ __forceinline__ float2 e2m1x2_to_float2(uint32_t byte) {
  uint32_t h2;
  asm("{ .reg .b8 lo, hi; mov.b16 {lo, hi}, %1; cvt.rn.f16x2.e2m1x2 %0, lo; }" : "=r"(h2) : "h"((unsigned short)byte));
  return __half22float2(*reinterpret_cast<const __half2*>(&h2));
}

// The eight codes of a word as floats, exact.
__device__ __forceinline__ void e2m1x8_to_float(uint32_t w, float* f) {
  uint32_t h[4];
  asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %4;\n"
      "cvt.rn.f16x2.e2m1x2 %0, b0; cvt.rn.f16x2.e2m1x2 %1, b1; cvt.rn.f16x2.e2m1x2 %2, b2; cvt.rn.f16x2.e2m1x2 %3, b3; }"
      : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3]) : "r"(w));
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 e = __half22float2(*reinterpret_cast<const __half2*>(&h[i]));
    f[2 * i] = e.x;
    f[2 * i + 1] = e.y;
  }
}

// eight floats by one 32-byte load (volatile: behind the wait for the kernel that writes them)
__device__ __forceinline__ void load8_wide(const float* p, float* f) {
  asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7]) : "l"(p));
}

// The same product along the tiled scale layout.  A 16-byte piece of that layout holds the scales of the rows l, l + 32,
// l + 64, l + 96 of a 128-row block for 4 blocks of 16 columns: a warp takes these four rows, lane k of it every 32nd block
// from k on, so that one 16-byte read of scales (shared by four lanes) and the 16 floats of v (which stay in L1) serve
// four rows.  With too few rows to fill the SMs that way, two or four warps (`split`) share the four rows: each takes every
// split-th round of 32 blocks and parks the block sums in shared memory; the lanes' sums are formed from there in order.
// The additions are those of the other kernels, in the same order: 16 products of a block one after the other, a lane's
// blocks one after the other, then the lanes pairwise, so which kernel runs does not show in the result (a sum that
// differs in its last bit can flip the rounding of an activation, and a block of decoder layers makes 1 % of that).
// Bound by issue, the conversions (two codes become two halves with one, exactly) and L1: a lane reads the 16 floats of its own
// block of v, so a warp's load of them touches 16 lines whatever its width, and with 32-byte loads (v on such a boundary) it does
// so twice instead of four times.  18944 x 3584 takes 11.9 us, its bytes 6.  Six weights in turn, us, gemv_staged_kernel or
// gemv_kernel / 16-byte loads / 32-byte loads, two rows' additions packed: 18944 x 3584 20.5 / 13.5 / 11.9, 3584 x 18944
// 23.6 / 17.8 / 17.0, 14336 x 4096 21.5 / 13.3 / 11.9, 4096 x 14336 18.5 / 14.5 / 13.2, 8960 x 1536 10.2 / 4.2 / 3.7,
// 1536 x 8960 7.7 / 5.6 / 5.3, 4096 x 4096 6.4 / 5.6 / 5.3.  (Packed additions where warps share rows: 4096 x 14336 13.7; the next
// round's codes in registers ahead of the work: 18944 x 3584 13.5.)  Four warps in a CTA: with eight the last ones end less evenly
// (3584 x 18944 19.0); a warp per two rows reads v and the scales twice (30).
constexpr int kGemvWarps = 4, kGemvCtasPerSm = 8;
// kWideV: v starts on a 32-byte boundary
template <bool kSplit, bool kWideV>
__global__ void __launch_bounds__(32 * kGemvWarps, kGemvCtasPerSm)
gemv_quad_kernel(const uint8_t* __restrict__ codes, const uint8_t* __restrict__ scales, const float* __restrict__ unit_ptr,
                 int64_t R, int64_t C, int trips, int split, const float* __restrict__ v, float* __restrict__ out) {
  extern __shared__ uint32_t s_sums[];                    // kSplit, per four rows: [5][trips][32], the sums of four rows and their scales
  grid_dependency_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int local = kSplit ? warp / split : warp, share = kSplit ? warp - local * split : 0;
  const int64_t quad = (int64_t)blockIdx.x * (kSplit ? kGemvWarps / split : kGemvWarps) + local;
  const int64_t row0 = (quad >> 5) * 128 + (quad & 31);   // this warp's rows: row0 + 32 c
  if (!kSplit && row0 >= R) return;
  const int sf_cols = (int)(C >> 4);
  const uint2* row_codes[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) row_codes[c] = reinterpret_cast<const uint2*>(codes) + (row0 + 32 * c < R ? row0 + 32 * c : R - 1) * sf_cols;
  const uint8_t* row_scales = scales + (row0 < R ? quad >> 5 : 0) * sf_tiles_per_row(C) * 512 + (quad & 31) * 16 + (lane >> 2) * 512;
  uint32_t* sums = s_sums + (kSplit ? local * 5 * trips * 32 : 0) + lane;
  const int byte = 8 * (lane & 3);
  float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 2
  for (int t = share; t < trips; t += kSplit ? split : 1) {
    const int k = t * 32 + lane;
    if (k < sf_cols) {
      const uint4 sw = __ldg(reinterpret_cast<const uint4*>(row_scales + (int64_t)t * 8 * 512));
      uint2 w[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) w[c] = __ldg(row_codes[c] + k);
      float f[16];
      if constexpr (kWideV) {
        load8_wide(v + 16 * (int64_t)k, f);
        load8_wide(v + 16 * (int64_t)k + 8, f + 8);
      } else {
        const float4* v4 = reinterpret_cast<const float4*>(v) + 4 * (int64_t)k;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 q = __ldg(v4 + i);
          f[4 * i] = q.x; f[4 * i + 1] = q.y; f[4 * i + 2] = q.z; f[4 * i + 3] = q.w;
        }
      }
      const uint32_t s4[4] = {sw.x >> byte, sw.y >> byte, sw.z >> byte, sw.w >> byte};
      if constexpr (kSplit) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float e[16];
          e2m1x8_to_float(w[c].x, e);
          e2m1x8_to_float(w[c].y, e + 8);
          float part = 0.0f;
#pragma unroll
          for (int i = 0; i < 16; ++i) part = fmaf(e[i], f[i], part);
          sums[(c * trips + t) * 32] = __float_as_uint(part);
        }
        sums[(4 * trips + t) * 32] = __byte_perm(__byte_perm(s4[0], s4[1], 0x0040), __byte_perm(s4[2], s4[3], 0x0040), 0x5410);
      } else {
#pragma unroll
        for (int c = 0; c < 4; c += 2) {                    // two rows' chains to a packed instruction
          f32x2 part = 0ull;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float e0[8], e1[8];
            e2m1x8_to_float(h == 0 ? w[c].x : w[c].y, e0);
            e2m1x8_to_float(h == 0 ? w[c + 1].x : w[c + 1].y, e1);
#pragma unroll
            for (int i = 0; i < 8; ++i) part = fma2(pack2(e0[i], e1[i]), pack2(f[8 * h + i], f[8 * h + i]), part);
          }
          float p[2];
          split2(part, p[0], p[1]);
          acc[c] = fmaf(p[0], e4m3_to_float((uint8_t)s4[c]), acc[c]);
          acc[c + 1] = fmaf(p[1], e4m3_to_float((uint8_t)s4[c + 1]), acc[c + 1]);
        }
      }
    }
  }
  const float unit = __ldg(unit_ptr);
  if (kSplit) __syncthreads();
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (kSplit) {
      if (c % split != share) continue;                   // four warps: a row each
#pragma unroll 8
      for (int t = 0; t < trips; ++t) {
        if (t * 32 + lane < sf_cols)
          acc[c] = fmaf(__uint_as_float(sums[(c * trips + t) * 32]), e4m3_to_float((uint8_t)(sums[(4 * trips + t) * 32] >> (8 * c))), acc[c]);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    if (lane == 0 && row0 + 32 * c < R) out[row0 + 32 * c] = acc[c] * unit;
  }
}

// The same product for a tall matrix (12288 rows and more) that neither gemv_quad_kernel nor gemv_staged_kernel takes: mostly
// narrow ones, of either layout (gemv_kernel / this, us: 152064 x 128 47 / 25, 12288 x 64 4.8 / 2.9, 18944 x 496 7.5 / 5.4).  Two
// e2m1 codes become two halves with one cvt (exact), and the 16 floats of v for a lane's block stay in registers across the
// 4 rows of the warp (v otherwise costs 8 times the bytes of the codes in L1 traffic).  Shorter matrices keep gemv_kernel:
// with four rows per warp they would not fill the SMs.
constexpr int kGemvTallRows = 4;          // rows per warp
constexpr int64_t kGemvTallMinRows = 12288;
constexpr int64_t kGemvTileMinCols = 512;

__global__ void __launch_bounds__(256)
gemv_tall_kernel(const uint2* __restrict__ codes, const uint8_t* __restrict__ scales,
                 const float* __restrict__ unit_ptr, int32_t sf_layout, int64_t R, int64_t C,
                 const float* __restrict__ v, float* __restrict__ out) {
  grid_dependency_wait();
  const int lane = threadIdx.x & 31;
  const int64_t row0 = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * kGemvTallRows;
  if (row0 >= R) return;
  const int64_t sf_cols = C >> 4;                          // blocks per row
  const int64_t tiles = sf_tiles_per_row(C);
  float acc[kGemvTallRows];
#pragma unroll
  for (int j = 0; j < kGemvTallRows; ++j) acc[j] = 0.0f;
  for (int64_t k = lane; k < sf_cols; k += 32) {
    float f[16];
    const float4* v4 = reinterpret_cast<const float4*>(v + k * 16);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 q = __ldg(v4 + i);
      f[4 * i] = q.x; f[4 * i + 1] = q.y; f[4 * i + 2] = q.z; f[4 * i + 3] = q.w;
    }
#pragma unroll
    for (int j = 0; j < kGemvTallRows; ++j) {
      const int64_t row = row0 + j;
      if (row >= R) break;                                 // uniform over the warp
      const uint2 w2 = __ldg(codes + row * sf_cols + k);
      const int64_t off = (sf_layout == METIS_SF_MMA) ? sf_mma_offset(row, k, tiles) : row * sf_cols + k;
      const float sc = e4m3_to_float(__ldg(scales + off));
      const uint32_t w[2] = {w2.x, w2.y};
      float part = 0.0f;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const float2 c = e2m1x2_to_float2((w[b >> 2] >> (8 * (b & 3))) & 0xFFu);
        part = fmaf(c.x, f[2 * b], part);
        part = fmaf(c.y, f[2 * b + 1], part);
      }
      acc[j] = fmaf(part, sc, acc[j]);
    }
  }
  const float unit = __ldg(unit_ptr);
#pragma unroll
  for (int j = 0; j < kGemvTallRows; ++j) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
    if (lane == 0 && row0 + j < R) out[row0 + j] = acc[j] * unit;
  }
}

// The same product with the vector staged in shared memory once per CTA and shared by all its rows: a CTA
// takes 8 * kRowsPerWarp consecutive rows and the whole of C, a warp kRowsPerWarp of them, a lane the blocks
// lane, lane + 32, ...  From global memory a block then costs its 8 bytes of codes and its scale byte; the 64
// bytes of v come from shared memory (stored chunk-major, so the lanes' 16-byte reads are conflict free) and are
// used for every row of the warp.  gemv_kernel reads v through L1 once per row: 8 times the bytes of the
// codes, which is what bounds it on wide matrices (3584 x 18944: 50 us; here 10).  Codes become floats by the
// hardware conversion, two per instruction.
constexpr int64_t kGemvStagedMaxCols = 40960;           // 160 KiB of v
constexpr int64_t kGemvStagedMinCols = 2048;
template <int kRowsPerWarp>
__global__ void __launch_bounds__(256)
gemv_staged_kernel(const uint2* __restrict__ codes, const uint8_t* __restrict__ scales,
                   const float* __restrict__ unit_ptr, int32_t sf_layout, int64_t R, int64_t C,
                   const float* __restrict__ v, float* __restrict__ out) {
  extern __shared__ float4 s_v[];                          // [4][sf_cols]: chunk j of block k at j * sf_cols + k
  grid_dependency_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sf_cols = (int)(C >> 4);                       // blocks per row
  const int64_t tiles = sf_tiles_per_row(C);
  for (int i = threadIdx.x; i < sf_cols * 4; i += 256)     // coalesced read of v, scattered 16-byte writes
    s_v[(i & 3) * sf_cols + (i >> 2)] = __ldg(reinterpret_cast<const float4*>(v) + i);
  __syncthreads();
  const int64_t row0 = ((int64_t)blockIdx.x * 8 + warp) * kRowsPerWarp;
  if (row0 >= R) return;
  float acc[kRowsPerWarp];
#pragma unroll
  for (int j = 0; j < kRowsPerWarp; ++j) acc[j] = 0.0f;
#pragma unroll(kRowsPerWarp == 1 ? 4 : 2)
  for (int k = lane; k < sf_cols; k += 32) {
    uint2 w2[kRowsPerWarp];
    uint32_t sb[kRowsPerWarp];
#pragma unroll
    for (int j = 0; j < kRowsPerWarp; ++j) {               // every global load of the trip before the arithmetic
      const int64_t row = row0 + j < R ? row0 + j : R - 1;
      w2[j] = __ldg(codes + row * sf_cols + k);
      const int64_t off = (sf_layout == METIS_SF_MMA) ? sf_mma_offset(row, k, tiles) : row * sf_cols + k;
      sb[j] = __ldg(scales + off);
    }
    float f[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 q = s_v[i * sf_cols + k];
      f[4 * i] = q.x; f[4 * i + 1] = q.y; f[4 * i + 2] = q.z; f[4 * i + 3] = q.w;
    }
#pragma unroll
    for (int j = 0; j < kRowsPerWarp; ++j) {
      const uint32_t w[2] = {w2[j].x, w2[j].y};
      float part = 0.0f;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const float2 c = e2m1x2_to_float2((w[b >> 2] >> (8 * (b & 3))) & 0xFFu);
        part = fmaf(c.x, f[2 * b], part);
        part = fmaf(c.y, f[2 * b + 1], part);
      }
      acc[j] = fmaf(part, e4m3_to_float((uint8_t)sb[j]), acc[j]);
    }
  }
  const float unit = __ldg(unit_ptr);
#pragma unroll
  for (int j = 0; j < kRowsPerWarp; ++j) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
    if (lane == 0 && row0 + j < R) out[row0 + j] = acc[j] * unit;
  }
}

// Few, wide rows (the rank-r factor V against a wide activation mean): one row per CTA, its blocks dealt round
// robin to all 256 threads, the eight warps' sums added in warp order.
__global__ void __launch_bounds__(256)
gemv_row_kernel(const uint2* __restrict__ codes, const uint8_t* __restrict__ scales,
                const float* __restrict__ unit_ptr, int32_t sf_layout, int64_t R, int64_t C,
                const float* __restrict__ v, float* __restrict__ out) {
  __shared__ float s_part[8];
  grid_dependency_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row = blockIdx.x;
  const int sf_cols = (int)(C >> 4);
  const int64_t tiles = sf_tiles_per_row(C);
  float acc = 0.0f;
#pragma unroll 2
  for (int k = threadIdx.x; k < sf_cols; k += 256) {
    const uint2 w2 = __ldg(codes + row * sf_cols + k);
    const int64_t off = (sf_layout == METIS_SF_MMA) ? sf_mma_offset(row, k, tiles) : row * sf_cols + k;
    const uint32_t sb = __ldg(scales + off);
    const float4* v4 = reinterpret_cast<const float4*>(v) + 4 * (int64_t)k;
    float f[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 q = __ldg(v4 + i);
      f[4 * i] = q.x; f[4 * i + 1] = q.y; f[4 * i + 2] = q.z; f[4 * i + 3] = q.w;
    }
    const uint32_t w[2] = {w2.x, w2.y};
    float part = 0.0f;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const float2 c = e2m1x2_to_float2((w[b >> 2] >> (8 * (b & 3))) & 0xFFu);
      part = fmaf(c.x, f[2 * b], part);
      part = fmaf(c.y, f[2 * b + 1], part);
    }
    acc = fmaf(part, e4m3_to_float((uint8_t)sb), acc);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) s_part[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float sum = 0.0f;
#pragma unroll
    for (int w8 = 0; w8 < 8; ++w8) sum += s_part[w8];
    out[row] = sum * __ldg(unit_ptr);
  }
}

template <int kRowsPerWarp>
static cudaError_t launch_gemv_staged(const uint2* codes, const uint8_t* scales, const float* unit, int32_t sf_layout,
                                      int64_t R, int64_t C, const float* v, float* out, cudaStream_t st) {
  auto kern = gemv_staged_kernel<kRowsPerWarp>;
  const size_t smem = (size_t)C * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  return launch_overlapped(kLaunchShort, kern, dim3((unsigned)ceil_div(R, 8 * kRowsPerWarp)), dim3(256), smem, st,
                           codes, scales, unit, sf_layout, R, C, v, out);
}

// How many warps share four rows: as many as bring an SM to 24 warps (12 to 15 run at 0.88 of the rate: 4096 x 4096 5.5 us
// with 28, 6.2 with 14), unless the rounds that the last warps lack cost as much (8960 x 1536 has three rounds: 4.4 us with
// a warp per four rows, 5.6 with two) or there are two rounds only, of which each warp would then have one (8960 x 768
// 3.2 us with a warp per four rows, 4.2 with two; 13038 x 560 3.9 / 5.8); below 8 warps always.  The block sums of eight CTAs
// have to leave room for v in L1.
constexpr int64_t kGemvWarpsPerSm = 24, kGemvFewWarpsPerSm = 8, kGemvL1Bytes = 208 << 10, kGemvSumBytesMax = 96 << 10;
static int64_t gemv_sum_bytes(int64_t C, int split) { return kGemvWarps / split * ceil_div(C, 512) * 5 * 32 * (int64_t)sizeof(float); }
static int gemv_split(int64_t R, int64_t C) {
  const int64_t sms = device_sm_count(), quads = ceil_div(R, 128) * 32, trips = ceil_div(C, 512);
  auto padded = [&](int k) { return ceil_div(trips, k) * k; };              // rounds, the missing ones of the last included
  int split = 1;
  auto sharing_pays = [&] {
    if (quads * split < sms * kGemvFewWarpsPerSm) return true;
    return trips > 2 && quads * split < sms * kGemvWarpsPerSm && padded(2 * split) * 10 <= padded(split) * 11;
  };
  while (split < kGemvWarps && trips >= 2 * split && sharing_pays()) split *= 2;
  while (split > 1 && split < kGemvWarps && kGemvCtasPerSm * gemv_sum_bytes(C, split) + C * (int64_t)sizeof(float) > kGemvL1Bytes) split *= 2;
  return gemv_sum_bytes(C, split) > kGemvSumBytesMax ? 1 : split;
}

// Whether gemv_quad_kernel is the faster one for a matrix in the tiled layout.  Against gemv_staged_kernel (staged -> quad, us):
// - from 8192 columns on, where that one fits two CTAs on an SM at most: always (2048 x 8192 7.0 -> 6.0, 8976 x 8192
//   22.5 -> 18.0, 12288 x 12288 38.9 -> 32.2);
// - where that one would give four rows to a warp: always (18944 x 3584 20.5 -> 13.5);
// - between: seven rounds or more (3584 x 3584 5.7 -> 5.1; 3072 x 3072 4.4 -> 5.0, 2048 x 2048 2.9 -> 3.15), up to 15 warps per
//   SM of four rows each, less than a quarter of the rounds missing (4608 x 5120 8.6 -> 7.7, 8192 x 4096 10.0 -> 9.6; but
//   10240 x 6432 18.5 -> 19.8, 3072 x 6432 7.1 -> 7.8); where warps share rows only to bring an SM to 24 of them, up to 14 and a
//   twentieth (6144 x 6144 12.3 -> 10.6; but 5816 x 5600 9.0 -> 10.0, 8357 x 5600 11.2 -> 12.2, 8357 x 4096 9.0 -> 9.4).
// Below 2048 columns it replaces gemv_kernel (8960 x 1536 10.2 -> 4.3, 4096 x 768 4.0 -> 3.2, 1024 x 1792 4.3 -> 2.7), except for
// few rows of two or three rounds (1024 x 768 2.1 -> 2.6, 2048 x 1024 2.7 -> 2.9, 3072 x 1024 3.4 -> 3.1).
static bool gemv_quad_wins(int64_t R, int64_t C) {
  if (C < kGemvStagedMinCols) return R >= (C > 512 && C <= 1536 ? 2560 : 512);
  if (R < 1024) return false;                                               // 512 x 3584: 3.5 -> 4.3
  const int64_t sms = device_sm_count(), split = gemv_split(R, C);
  if (C >= 8192 || ceil_div(R, 32) >= 3 * sms) return true;
  const int64_t quads = ceil_div(R, 128) * 32, columns = ceil_div(ceil_div(C, 512), split) * split * 512;   // missing ones included
  if (split > 1 && quads >= kGemvFewWarpsPerSm * sms && (quads >= 14 * sms || columns * 20 > 21 * C)) return false;
  return C >= 3584 && quads < 15 * sms && columns * 4 < 5 * C;
}

static cudaError_t launch_gemv_quad(const uint8_t* codes, const uint8_t* scales, const float* unit, int64_t R, int64_t C,
                                    const float* v, float* out, cudaStream_t st) {
  const int64_t quads = ceil_div(R, 128) * 32, trips = ceil_div(C, 512);
  const int split = gemv_split(R, C);
  const dim3 grid((unsigned)ceil_div(quads * split, kGemvWarps)), block(32 * kGemvWarps);
  const bool wide_v = (reinterpret_cast<uintptr_t>(v) & 31u) == 0;
  if (split == 1)
    return launch_overlapped(kLaunchShort, wide_v ? gemv_quad_kernel<false, true> : gemv_quad_kernel<false, false>, grid, block, 0, st, codes, scales,
                             unit, R, C, (int)trips, 1, v, out);
  const size_t smem = (size_t)gemv_sum_bytes(C, split);
  auto kern = wide_v ? gemv_quad_kernel<true, true> : gemv_quad_kernel<true, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemvSumBytesMax);
  if (e != cudaSuccess) return e;
  return launch_overlapped(kLaunchShort, kern, grid, block, smem, st, codes, scales, unit, R, C, (int)trips, split, v, out);
}

// t = bf16( float(bf16(yv * s)) / (unit_a * unit_b) ), 8 elements per thread
template <typename TS>
__global__ void __launch_bounds__(256)
lowrank_scale_kernel(const __nv_bfloat16* __restrict__ yv, int64_t M, int64_t r, int64_t ld,
                     const TS* __restrict__ s, const float* __restrict__ unit_a,
                     const float* __restrict__ unit_b, __nv_bfloat16* __restrict__ t) {
  grid_dependency_wait();
  const int64_t groups_per_row = r >> 3;
  const float div = __fmul_rn(__ldg(unit_a), __ldg(unit_b));
  const bool small = M * groups_per_row < ((int64_t)1 << 31);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M * groups_per_row;
       i += (int64_t)gridDim.x * blockDim.x) {
    // 32-bit index arithmetic where it fits (a 64-bit division is a subroutine of ~100 instructions)
    const int64_t m = small ? (int64_t)((uint32_t)i / (uint32_t)groups_per_row) : i / groups_per_row;
    const int64_t j0 = (i - m * groups_per_row) * 8;
    const uint4 w = __ldg(reinterpret_cast<const uint4*>(yv + m * ld + j0));
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
    uint32_t out[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      __nv_bfloat162 s2;
      if constexpr (sizeof(TS) == 2) s2 = *reinterpret_cast<const __nv_bfloat162*>(s + j0 + 2 * k);
      else s2 = __floats2bfloat162_rn(__ldg(s + j0 + 2 * k), __ldg(s + j0 + 2 * k + 1));
      const __nv_bfloat162 ts = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&ww[k]), s2);   // one rounding: the product is exact in fp32
      const uint32_t tw = *reinterpret_cast<const uint32_t*>(&ts);
      const __nv_bfloat162 o = __floats2bfloat162_rn(__fdiv_rn(bf16_lo(tw), div), __fdiv_rn(bf16_hi(tw), div));
      out[k] = *reinterpret_cast<const uint32_t*>(&o);
    }
    *reinterpret_cast<uint4*>(t + m * r + j0) = make_uint4(out[0], out[1], out[2], out[3]);
  }
}

// The rank-r factors of an fp32 layer as bf16 operands of the side product, both in one launch: t32 = (yv * s) / (unit_a * unit_b)
// and u, either rounded (kParts = 1) or split into a bf16 head and tail, [Th Tl Th] and [Uh Uh Ul] (kParts = 3).  One element
// per thread and round: the operands are a few hundred KB, and what it replaced were a dozen launches of one operation
// each (issued from Python 85 us of host time, 25 on the GPU at 2048 x 64; now 12 and 3).
template <typename TS, int kParts>
__global__ void __launch_bounds__(256)
lowrank_factors_kernel(const float* __restrict__ yv, int64_t M, int64_t r, int64_t ldy, const TS* __restrict__ s, const float* __restrict__ unit_a,
                       const float* __restrict__ unit_b, __nv_bfloat16* __restrict__ t, const float* __restrict__ u, int64_t N, int64_t ldu,
                       __nv_bfloat16* __restrict__ u_out) {
  grid_dependency_wait();
  const float units = __fmul_rn(__ldg(unit_a), __ldg(unit_b));
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (M + N) * r; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / r, col = i - row * r;
    const bool of_t = row < M;
    float v;
    if (of_t) {
      float sv;
      if constexpr (sizeof(TS) == 2) sv = __bfloat162float(s[col]); else sv = s[col];
      v = __fdiv_rn(__fmul_rn(yv[row * ldy + col], sv), units);
    } else {
      v = u[(row - M) * ldu + col];
    }
    const __nv_bfloat16 head = __float2bfloat16_rn(v);
    __nv_bfloat16* to = (of_t ? t + row * (kParts * r) : u_out + (row - M) * (kParts * r)) + col;
    to[0] = head;
    if constexpr (kParts == 3) {
      const __nv_bfloat16 tail = __float2bfloat16_rn(__fsub_rn(v, __bfloat162float(head)));
      to[r] = of_t ? tail : head;
      to[2 * r] = of_t ? head : tail;
    }
  }
}

}  // namespace metis

using namespace metis;

extern "C" int32_t metis_lowrank_scale(const void* yv, int64_t M, int64_t r, int64_t ld, const void* s,
                                       int32_t s_dtype, const float* unit_a, const float* unit_b, void* t,
                                       void* stream) {
  if (!yv || !s || !unit_a || !unit_b || !t) return fail(METIS_ERR_BAD_ARGUMENT, "null pointer");
  if (M <= 0 || r <= 0 || r % 8 != 0) return fail(METIS_ERR_BAD_SHAPE, "bad shape [%lld, %lld]: r must be a positive multiple of 8", (long long)M, (long long)r);
  if (s_dtype != METIS_DTYPE_BF16 && s_dtype != METIS_DTYPE_F32) return fail(METIS_ERR_BAD_ARGUMENT, "unknown s_dtype %d", s_dtype);
  if (ld < r || ld % 8 != 0 || !aligned16(yv) || !aligned16(t) || (reinterpret_cast<uintptr_t>(s) & 3u))
    return fail(METIS_ERR_BAD_ALIGNMENT, "yv and t must be 16-byte aligned, ld a multiple of 8 and >= r");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int64_t blocks = ceil_div(M * (r >> 3), 256);
  const int64_t cap = (int64_t)device_sm_count() * 16;
  if (blocks > cap) blocks = cap;
  const __nv_bfloat16* y = static_cast<const __nv_bfloat16*>(yv);
  __nv_bfloat16* o = static_cast<__nv_bfloat16*>(t);
  if (s_dtype == METIS_DTYPE_BF16)
    launch_overlapped(kLaunchShort, lowrank_scale_kernel<__nv_bfloat16>, dim3((unsigned)blocks), dim3(256), 0, st, y, M, r, ld, static_cast<const __nv_bfloat16*>(s), unit_a, unit_b, o);
  else
    launch_overlapped(kLaunchShort, lowrank_scale_kernel<float>, dim3((unsigned)blocks), dim3(256), 0, st, y, M, r, ld, static_cast<const float*>(s), unit_a, unit_b, o);
  METIS_CUDA_OK(cudaGetLastError());
  return METIS_OK;
}

extern "C" int32_t metis_lowrank_factors(const float* yv, int64_t M, int64_t r, int64_t ldy, const void* s, int32_t s_dtype,
                                         const float* unit_a, const float* unit_b, void* t, const float* u, int64_t N, int64_t ldu,
                                         void* u_out, int32_t parts, void* stream) {
  if (!yv || !s || !unit_a || !unit_b || !t || !u || !u_out) return fail(METIS_ERR_BAD_ARGUMENT, "null pointer");
  if (M <= 0 || N <= 0 || r <= 0 || ldy < r || ldu < r) return fail(METIS_ERR_BAD_SHAPE, "bad shape [%lld, %lld], [%lld, %lld]", (long long)M, (long long)r, (long long)N, (long long)r);
  if (s_dtype != METIS_DTYPE_BF16 && s_dtype != METIS_DTYPE_F32) return fail(METIS_ERR_BAD_ARGUMENT, "unknown s_dtype %d", s_dtype);
  if (parts != 1 && parts != 3) return fail(METIS_ERR_BAD_ARGUMENT, "parts must be 1 or 3");
  int64_t blocks = ceil_div((M + N) * r, 256);
  if (blocks > (int64_t)device_sm_count() * 16) blocks = (int64_t)device_sm_count() * 16;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  auto run = [&](auto kern, auto* sv) {
    return launch_overlapped(kLaunchShort, kern, dim3((unsigned)blocks), dim3(256), 0, st, yv, M, r, ldy, sv, unit_a, unit_b, static_cast<__nv_bfloat16*>(t), u, N,
                             ldu, static_cast<__nv_bfloat16*>(u_out));
  };
  const __nv_bfloat16* s16 = static_cast<const __nv_bfloat16*>(s);
  const float* s32 = static_cast<const float*>(s);
  METIS_CUDA_OK(s_dtype == METIS_DTYPE_BF16 ? (parts == 3 ? run(lowrank_factors_kernel<__nv_bfloat16, 3>, s16) : run(lowrank_factors_kernel<__nv_bfloat16, 1>, s16))
                                            : (parts == 3 ? run(lowrank_factors_kernel<float, 3>, s32) : run(lowrank_factors_kernel<float, 1>, s32)));
  return METIS_OK;
}

static int32_t dequantize(const uint8_t* codes, const uint8_t* scales, const UnitPtrs unit, int32_t sf_layout, int64_t R, int64_t C,
                          const float* add_row_vec, void* out, int32_t out_dtype, int64_t ld, void* stream) {
  if (!codes || !scales || !unit.u0 || !out) return fail(METIS_ERR_BAD_ARGUMENT, "null pointer");
  if (R <= 0 || C <= 0 || C % 16 != 0) return fail(METIS_ERR_BAD_SHAPE, "bad shape [%lld, %lld]", (long long)R, (long long)C);
  if (sf_layout != METIS_SF_ROWMAJOR && sf_layout != METIS_SF_MMA) return fail(METIS_ERR_BAD_ARGUMENT, "unknown sf_layout %d", sf_layout);
  if (out_dtype != METIS_DTYPE_BF16 && out_dtype != METIS_DTYPE_F32) return fail(METIS_ERR_BAD_ARGUMENT, "unknown out_dtype %d", out_dtype);
  if (ld < C || ld % 8 != 0 || !aligned16(out) || !aligned16(codes))
    return fail(METIS_ERR_BAD_ALIGNMENT, "out and codes must be 16-byte aligned, ld a multiple of 8 and >= C");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int64_t total = R * (C >> 3);
  int64_t blocks = ceil_div(total, 256);
  const int64_t cap = (int64_t)device_sm_count() * 32;
  if (blocks > cap) blocks = cap;
  const uint32_t* c32 = reinterpret_cast<const uint32_t*>(codes);
  if (out_dtype == METIS_DTYPE_BF16)
    launch_overlapped(kLaunchShort, unit.u1 ? dequantize_kernel<__nv_bfloat16, true> : dequantize_kernel<__nv_bfloat16, false>, dim3((unsigned)blocks), dim3(256), 0, st, c32, scales, unit, sf_layout, R, C, add_row_vec, static_cast<__nv_bfloat16*>(out), ld);
  else
    launch_overlapped(kLaunchShort, unit.u1 ? dequantize_kernel<float, true> : dequantize_kernel<float, false>, dim3((unsigned)blocks), dim3(256), 0, st, c32, scales, unit, sf_layout, R, C, add_row_vec, static_cast<float*>(out), ld);
  METIS_CUDA_OK(cudaGetLastError());
  return METIS_OK;
}

extern "C" int32_t metis_nvfp4_dequantize(const uint8_t* codes, const uint8_t* scales, const float* unit,
                                          int32_t sf_layout, int64_t R, int64_t C,
                                          const float* add_row_vec, void* out, int32_t out_dtype,
                                          int64_t ld, void* stream) {
  return dequantize(codes, scales, UnitPtrs{unit, nullptr, nullptr, nullptr}, sf_layout, R, C, add_row_vec, out, out_dtype, ld, stream);
}

extern "C" int32_t metis_nvfp4_dequantize_ratio(const uint8_t* codes, const uint8_t* scales, const float* unit0, const float* unit1,
                                                const float* over0, const float* over1, int32_t sf_layout, int64_t R, int64_t C,
                                                void* out, int32_t out_dtype, int64_t ld, void* stream) {
  if (!unit1 || !over0 || !over1) return fail(METIS_ERR_BAD_ARGUMENT, "null pointer");
  return dequantize(codes, scales, UnitPtrs{unit0, unit1, over0, over1}, sf_layout, R, C, nullptr, out, out_dtype, ld, stream);
}

extern "C" int32_t metis_nvfp4_gemv(const uint8_t* codes, const uint8_t* scales, const float* unit,
                                    int32_t sf_layout, int64_t R, int64_t C, const float* v, float* out,
                                    void* stream) {
  if (!codes || !scales || !unit || !out) return fail(METIS_ERR_BAD_ARGUMENT, "null pointer");
  if (R <= 0 || C <= 0 || C % 16 != 0) return fail(METIS_ERR_BAD_SHAPE, "bad shape [%lld, %lld]", (long long)R, (long long)C);
  if (sf_layout != METIS_SF_ROWMAJOR && sf_layout != METIS_SF_MMA) return fail(METIS_ERR_BAD_ARGUMENT, "unknown sf_layout %d", sf_layout);
  if (!aligned16(codes)) return fail(METIS_ERR_BAD_ALIGNMENT, "codes must be 16-byte aligned");
  if (v && !aligned16(v)) return fail(METIS_ERR_BAD_ALIGNMENT, "v must be 16-byte aligned");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const uint2* c4 = reinterpret_cast<const uint2*>(codes);
  // The kernel along the tiled scales where that is the layout and it is the faster one (the bits are the same).
  const bool tiled = sf_layout == METIS_SF_MMA && aligned16(scales) && C >= kGemvTileMinCols && C < ((int64_t)1 << 31);
  // Otherwise, rows of 2048 elements and more: the kernel that stages v in shared memory; too few rows for it: a CTA per
  // row.  Every CTA stages the whole of v, so with very wide rows fewer CTAs of more rows win although they
  // fill the SMs less evenly (3584 x 18944: 16 rows per CTA 19.6 us, 8 rows 28.2).
  if (v && tiled && gemv_quad_wins(R, C)) {
    METIS_CUDA_OK(launch_gemv_quad(codes, scales, unit, R, C, v, out, st));
  } else if (v && C >= kGemvStagedMinCols && C <= kGemvStagedMaxCols) {
    const int64_t sms = device_sm_count();
    const bool wide = C >= 8192;
    const int64_t want = wide ? sms : 3 * sms;               // CTAs a launch should at least have
    if (ceil_div(R, 32) >= want) METIS_CUDA_OK(launch_gemv_staged<4>(c4, scales, unit, sf_layout, R, C, v, out, st));
    else if (ceil_div(R, 16) >= want) METIS_CUDA_OK(launch_gemv_staged<2>(c4, scales, unit, sf_layout, R, C, v, out, st));
    else if (R >= (wide ? 4 * sms : want)) METIS_CUDA_OK(launch_gemv_staged<1>(c4, scales, unit, sf_layout, R, C, v, out, st));
    else METIS_CUDA_OK(launch_overlapped(kLaunchShort, gemv_row_kernel, dim3((unsigned)R), dim3(256), 0, st, c4, scales, unit, sf_layout, R, C, v, out));
  } else if (v && R >= kGemvTallMinRows) launch_overlapped(kLaunchShort, gemv_tall_kernel, dim3((unsigned)ceil_div(R, 8 * kGemvTallRows)), dim3(256), 0, st, c4, scales, unit, sf_layout, R, C, v, out);
  else if (v) launch_overlapped(kLaunchShort, gemv_kernel<true>, dim3((unsigned)ceil_div(R, 8)), dim3(256), 0, st, c4, scales, unit, sf_layout, R, C, v, out);
  else   launch_overlapped(kLaunchShort, gemv_kernel<false>, dim3((unsigned)ceil_div(R, 8)), dim3(256), 0, st, c4, scales, unit, sf_layout, R, C, v, out);
  METIS_CUDA_OK(cudaGetLastError());
  return METIS_OK;
}

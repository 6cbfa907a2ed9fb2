// Fused RMSNorm -> NVFP4 quantizer: every activation row is read from HBM exactly once.
//
// A CTA of 256 threads owns one row at a time (persistent loop over rows).  Each thread keeps
// up to kChunks groups of 8 elements in registers, the CTA reduces the sum of squares, and
// the normalised, gamma-scaled row is quantized straight from registers: two neighbouring
// lanes form a 16-element block exactly as in the stand-alone quantizer.  The E4M3 scale
// bytes are produced by the shared finalisation pass (they need the tensor-wide maximum).
#include "common.cuh"
#include "tma.cuh"

namespace metis {

constexpr int kNormThreads = 256;

// Rounds two floats to bf16 and back (one packed conversion).
__device__ __forceinline__ void round_bf16x2(float& a, float& b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  const uint32_t w = *reinterpret_cast<const uint32_t*>(&h);
  a = bf16_lo(w);
  b = bf16_hi(w);
}

// A CTA is bx x by threads: bx threads (a power of two, or a multiple of 32) share a row, each owning kBlocks
// 16-element blocks tx, tx + bx, ...; by rows are in flight per CTA.  Row sums of squares are
// reduced with shuffles inside a warp and through shared memory across the warps of a row.
template <typename TX, typename TG, int kBlocks, bool kWriteNorm>
__global__ void __launch_bounds__(kNormThreads)
rmsnorm_quantize_kernel(const TX* __restrict__ x, int rows, int blocks_per_row, int64_t ld,
                        const TG* __restrict__ gamma, float eps, uint2* __restrict__ codes,
                        float* __restrict__ amax_out, unsigned int* __restrict__ gmax,
                        unsigned int* __restrict__ records, void* __restrict__ norm_out) {
  grid_dependency_wait();
  // The product normalised(x) * gamma has the promoted dtype: bf16 only if both are bf16.
  constexpr bool kProductBf16 = (sizeof(TX) == 2) && (sizeof(TG) == 2);
  __shared__ float s_red[kNormThreads / 32];
  __shared__ float s_rs[kNormThreads / 32];        // reciprocal RMS of each row in flight (rows span >= 1 warp here)
  const int bx = blockDim.x, by = blockDim.y;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int tid = ty * bx + tx;
  const int lane = tid & 31, warp = tid >> 5;
  const int seg = bx < 32 ? bx : 32;                 // lanes of one row inside a warp
  const int warps_per_row = bx >> 5;                 // 0 when a warp holds several rows
  const float n_cols = (float)(blocks_per_row * 16);
  float running = 0.0f;

  // The row after the current one is already on its way from HBM while the current one is reduced,
  // normalised and quantized: its blocks wait in registers as loaded.
  RawBlock<TX> raw[kBlocks];
  auto fetch = [&](int r_first) {
    const int r = r_first + ty;
#pragma unroll
    for (int j = 0; j < kBlocks; ++j) {
      const int bc = tx + j * bx;
      if (r < rows && bc < blocks_per_row) raw[j].load(x + (int64_t)r * ld + (int64_t)bc * 16);
    }
  };
  fetch(blockIdx.x * by);

  for (int r0 = blockIdx.x * by; r0 < rows; r0 += gridDim.x * by) {
    const int r = r0 + ty;
    const bool row_live = r < rows;
    float v[kBlocks][16];
    float ss = 0.0f;
#pragma unroll
    for (int j = 0; j < kBlocks; ++j) {
      const int bc = tx + j * bx;
      if (row_live && bc < blocks_per_row) {
        raw[j].unpack(v[j]);
#pragma unroll
        for (int i = 0; i < 16; ++i) ss = __fmaf_rn(v[j][i], v[j][i], ss);
      }
    }
    fetch(r0 + gridDim.x * by);
    for (int o = seg >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    // x * rsqrt(mean(x^2) + eps) with the IEEE operations the CPU reference uses: correctly
    // rounded division, square root and reciprocal (llama.py:23-24).  The sequence is some 50
    // instructions, so one thread per row runs it and the others pick the result up.
    float rs;
    if (warps_per_row > 1) {                           // uniform over the CTA
      if (lane == 0) s_red[warp] = ss;
      __syncthreads();
      if (tx == 0) {
        float tot = 0.0f;
        for (int w = 0; w < warps_per_row; ++w) tot += s_red[ty * warps_per_row + w];
        s_rs[ty] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, n_cols), eps)));
      }
      __syncthreads();                                 // also: s_red may be rewritten by the next row
      rs = s_rs[ty];
    } else {
      rs = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, n_cols), eps)));   // every lane of the row holds the sum
    }

#pragma unroll
    for (int j = 0; j < kBlocks; ++j) {
      const int bc = tx + j * bx;
      if (!(row_live && bc < blocks_per_row)) continue;
      float y[16];
      float a;
      if constexpr (kProductBf16) {
        // both roundings of the reference in packed bf16: n = bf16(x * rs) (llama.py:28), then
        // n * gamma as one bf16x2 multiply: the product of two bf16 is exact in fp32, so rounding
        // it once to bf16 is what the fp32 multiply followed by the conversion gives (llama.py:31)
        RawBlock<__nv_bfloat16> graw;
        graw.load(reinterpret_cast<const __nv_bfloat16*>(gamma) + (int64_t)bc * 16);
        const uint32_t gw[8] = {graw.a.x, graw.a.y, graw.a.z, graw.a.w, graw.b.x, graw.b.y, graw.b.z, graw.b.w};
        const f32x2 rs2 = pack2(rs, rs);
        __nv_bfloat162 amax2 = __floats2bfloat162_rn(0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float n0, n1;
          split2(mul2(pack2(v[j][2 * i], v[j][2 * i + 1]), rs2), n0, n1);
          const __nv_bfloat162 n2 = __floats2bfloat162_rn(n0, n1);
          const __nv_bfloat162 p2 = __hmul2(n2, *reinterpret_cast<const __nv_bfloat162*>(&gw[i]));
          amax2 = __hmax2(amax2, __habs2(p2));
          const uint32_t w = *reinterpret_cast<const uint32_t*>(&p2);
          y[2 * i] = bf16_lo(w);
          y[2 * i + 1] = bf16_hi(w);
        }
        const uint32_t aw = *reinterpret_cast<const uint32_t*>(&amax2);
        a = fmaxf(bf16_lo(aw), bf16_hi(aw));
      } else {
        float g[16];
        Load16<TG>::load(gamma + (int64_t)bc * 16, g);
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          float n0 = __fmul_rn(v[j][i], rs), n1 = __fmul_rn(v[j][i + 1], rs);
          if (sizeof(TX) == 2) round_bf16x2(n0, n1);                      // .type_as(x), llama.py:28
          y[i] = __fmul_rn(n0, g[i]);                                     // * weight, llama.py:31
          y[i + 1] = __fmul_rn(n1, g[i + 1]);
        }
        a = abs_max16(y);
      }
      uint32_t packed[2];
      quantize_rn<2>(y, block_scale_from_amax(a), packed);
      const int64_t b = (int64_t)r * blocks_per_row + bc;
      codes[b] = make_uint2(packed[0], packed[1]);
      amax_out[b] = a;
      running = fmaxf(running, a);
      if (kWriteNorm) {
        if (kProductBf16) {
          __nv_bfloat162 o[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = __floats2bfloat162_rn(y[2 * i], y[2 * i + 1]);   // exact: already bf16 values
          uint4* dst = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(norm_out) + b * 16);
          dst[0] = reinterpret_cast<uint4*>(o)[0];
          dst[1] = reinterpret_cast<uint4*>(o)[1];
        } else {
          float4* dst = reinterpret_cast<float4*>(static_cast<float*>(norm_out) + b * 16);
#pragma unroll
          for (int i = 0; i < 4; ++i) dst[i] = make_float4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]);
        }
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) running = fmaxf(running, __shfl_xor_sync(0xffffffffu, running, o));
  if (!records) {
    if (lane == 0 && running > 0.0f) atomicMax(gmax, __float_as_uint(running));
    return;
  }
  // a record per CTA: nobody has to zero a shared maximum first
  __shared__ float s_top[kNormThreads / 32];
  if (lane == 0) s_top[warp] = running;
  __syncthreads();
  if (tid == 0) {
    float top = 0.0f;
    for (int w = 0; w < (bx * by + 31) / 32; ++w) top = fmaxf(top, s_top[w]);
    records[3 * blockIdx.x] = __float_as_uint(top);
    records[3 * blockIdx.x + 1] = 0u;
    records[3 * blockIdx.x + 2] = 0u;
    if (blockIdx.x == 0) records[-1] = gridDim.x;
  }
}

// ---- decode-sized inputs: one launch ---------------------------------------------------------------
// The same row arithmetic for a handful of rows, run as ONE thread-block cluster of up to 8 CTAs: a CTA
// of bx x by = 512 threads takes up to kNormSmallPasses groups of `by` rows, every block maximum stays in a
// register, the tensor-wide maximum crosses the cluster through shared memory, and the threads write
// their own E4M3 bytes: no scale pass, no scratch in global memory.

// normalised(x) * gamma for one 16-element block, with the reference's roundings (llama.py:28, 31);
// returns the block maximum.
template <typename TX, typename TG>
__device__ __forceinline__ float norm_block(const float (&v)[16], float rs, const TG* __restrict__ gamma16, float (&y)[16]) {
  constexpr bool kProductBf16 = (sizeof(TX) == 2) && (sizeof(TG) == 2);
  if constexpr (kProductBf16) {
    RawBlock<__nv_bfloat16> graw;
    graw.load(reinterpret_cast<const __nv_bfloat16*>(gamma16));
    const uint32_t gw[8] = {graw.a.x, graw.a.y, graw.a.z, graw.a.w, graw.b.x, graw.b.y, graw.b.z, graw.b.w};
    const f32x2 rs2 = pack2(rs, rs);
    __nv_bfloat162 amax2 = __floats2bfloat162_rn(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float n0, n1;
      split2(mul2(pack2(v[2 * i], v[2 * i + 1]), rs2), n0, n1);
      const __nv_bfloat162 n2 = __floats2bfloat162_rn(n0, n1);
      const __nv_bfloat162 p2 = __hmul2(n2, *reinterpret_cast<const __nv_bfloat162*>(&gw[i]));
      amax2 = __hmax2(amax2, __habs2(p2));
      const uint32_t w = *reinterpret_cast<const uint32_t*>(&p2);
      y[2 * i] = bf16_lo(w);
      y[2 * i + 1] = bf16_hi(w);
    }
    const uint32_t aw = *reinterpret_cast<const uint32_t*>(&amax2);
    return fmaxf(bf16_lo(aw), bf16_hi(aw));
  } else {
    float g[16];
    Load16<TG>::load(gamma16, g);
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
      float n0 = __fmul_rn(v[i], rs), n1 = __fmul_rn(v[i + 1], rs);
      if (sizeof(TX) == 2) round_bf16x2(n0, n1);
      y[i] = __fmul_rn(n0, g[i]);
      y[i + 1] = __fmul_rn(n1, g[i + 1]);
    }
    return abs_max16(y);
  }
}

// ---- long inputs, bf16 rows of up to 4096 elements: a warp per row --------------------------------------------
// With a CTA per row two barriers stand between its parts (3.1 of 10.5 stalled warps waited there, issue slots 66 % busy,
// 18 instructions per element).  A warp that owns its row needs none: the sum of squares goes through shuffles.  The sums are
// added in the order of the CTA-per-row kernel (16 squares of a block one after the other, lanes by butterfly, then the groups
// of 32 blocks in order), so the results are its results.  Loads that leave L2 first (to keep the block maxima there for the
// scale pass) change nothing here and cost the tile kernels of quantize.cu 20 %; a prefetch of the next row into L2 changes
// nothing either.
// Fewer rows do not fill the SMs with a warp each (both launches, a CTA / a warp per row, us): 896 x 4096 7.6 / 9.2, 640 x 3584
// 6.5 / 8.3, 640 x 2048 7.0 / 7.5, 800 x 2048 6.0 / 6.1; equal from 1024 x 3584 (9.5 / 9.6) on, and rows of 512 elements do not
// care (896: 4.9 / 4.5).
constexpr int64_t kNormRowsMinRows = 1024;

// Narrow rows, and wide ones where norm_rows_staged says so: the row stays in registers as loaded (kM blocks of 16 elements per lane, block lane + 32 j); two blocks' chains
// of squares share one packed instruction.
constexpr int kNormRowThreads = 256;
template <typename TG, int kM, bool kWriteNorm>
__global__ void __launch_bounds__(kNormRowThreads, kM <= 3 ? 3 : 2)
rmsnorm_quantize_rows_kernel(const __nv_bfloat16* __restrict__ x, int rows, int blocks_per_row, int64_t ld,
                             const TG* __restrict__ gamma, float eps, uint2* __restrict__ codes,
                             float* __restrict__ amax_out, unsigned int* __restrict__ gmax,
                             unsigned int* __restrict__ records, void* __restrict__ norm_out) {
  grid_dependency_wait();
  constexpr bool kProductBf16 = sizeof(TG) == 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float n_cols = (float)(blocks_per_row * 16);
  float running = 0.0f;
  const int row_step = gridDim.x * (kNormRowThreads / 32);
  for (int r = blockIdx.x * (kNormRowThreads / 32) + warp; r < rows; r += row_step) {
    const __nv_bfloat16* row = x + (int64_t)r * ld;
    RawBlock<__nv_bfloat16> raw[kM];
#pragma unroll
    for (int j = 0; j < kM; ++j) {
      raw[j].a = raw[j].b = make_uint4(0u, 0u, 0u, 0u);
      if (lane + 32 * j < blocks_per_row) raw[j].load(row + (lane + 32 * j) * 16);
    }
    float ss[kM];
#pragma unroll
    for (int j = 0; j < kM; j += 2) {
      float v[16], w[16];
      raw[j].unpack(v);
      if (j + 1 < kM) {
        raw[j + 1 < kM ? j + 1 : j].unpack(w);
        f32x2 acc = 0ull;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const f32x2 e = pack2(v[i], w[i]);
          acc = fma2(e, e, acc);
        }
        split2(acc, ss[j], ss[j + 1 < kM ? j + 1 : j]);
      } else {
        ss[j] = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i) ss[j] = __fmaf_rn(v[i], v[i], ss[j]);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int j = 0; j < kM; ++j) ss[j] += __shfl_xor_sync(0xffffffffu, ss[j], o);
    }
    float tot = 0.0f;
#pragma unroll
    for (int j = 0; j < kM; ++j) tot += ss[j];
    const float rs = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, n_cols), eps)));   // llama.py:23-24
#pragma unroll
    for (int j = 0; j < kM; ++j) {
      const int bc = lane + 32 * j;
      if (bc >= blocks_per_row) continue;
      float v[16], y[16];
      raw[j].unpack(v);
      const float a = norm_block<__nv_bfloat16, TG>(v, rs, gamma + bc * 16, y);
      uint32_t packed[2];
      quantize_rn<2>(y, block_scale_from_amax(a), packed);
      const int64_t b = (int64_t)r * blocks_per_row + bc;
      codes[b] = make_uint2(packed[0], packed[1]);
      amax_out[b] = a;
      running = fmaxf(running, a);
      if (kWriteNorm) {
        if (kProductBf16) {
          __nv_bfloat162 o[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = __floats2bfloat162_rn(y[2 * i], y[2 * i + 1]);   // exact: already bf16 values
          uint4* dst = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(norm_out) + b * 16);
          dst[0] = reinterpret_cast<uint4*>(o)[0];
          dst[1] = reinterpret_cast<uint4*>(o)[1];
        } else {
          float4* dst = reinterpret_cast<float4*>(static_cast<float*>(norm_out) + b * 16);
#pragma unroll
          for (int i = 0; i < 4; ++i) dst[i] = make_float4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]);
        }
      }
    }
  }
  const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(running));       // >= 0: the bits order like the value
  if (!records) {
    if (lane == 0 && top > 0u) atomicMax(gmax, top);
    return;
  }
  __shared__ unsigned s_top[kNormRowThreads / 32];
  if (lane == 0) s_top[warp] = top;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned m = 0u;
    for (int w = 0; w < kNormRowThreads / 32; ++w) m = max(m, s_top[w]);
    records[3 * blockIdx.x] = m;
    records[3 * blockIdx.x + 1] = 0u;
    records[3 * blockIdx.x + 2] = 0u;
    if (blockIdx.x == 0) records[-1] = gridDim.x;
  }
}

// Wider ones: one CTA per SM, whose lanes 0 fetch a warp's row into its part of shared memory by one bulk copy, and the next one
// as soon as the row has been read for the second time.  (In registers such a row takes 128 of them a thread, which leaves 16
// warps per SM, and a quarter of their time they waited for its loads.)  First reading: the sum of squares, by the
// multiply-add that takes bf16 operands.  Second: norm and quantization, block by block, in 64 registers.  The butterflies of
// the groups of 32 blocks share their shuffles.  Rows of whole 64-element groups are fetched with the 128-byte swizzle (one
// box of 64 x cols/64), which keeps both readings free of bank conflicts; others as they lie, at two wavefronts for one.
// Bound by issue (190 instructions per block of 16, 67 % of the slots at 65536 x 3584, 30 warps) and close to memory.  Both launches, row in registers /
// in shared memory, us: 65536 x 4096 191 / 150, x 3584 165 / 134, x 2048 101 / 78, x 1536 73 / 61, x 1024 52 / 44, 16384 x 3584
// 45 / 40, 1024 x 4096 9.4 / 7.8.  Narrow rows gain less, and few of them lose what setting the copies up costs (x 1024: 1024
// 5.3 / 5.5, 8192 9.6 / 10.1, 16384 17.7 / 16.8; x 768: 2048 6.0 / 6.3, 16384 17.5 / 16.0; x 512: 2048 4.8 / 5.2, 16384
// 10.0 / 11.0, 65536 30.1 / 29.6), so up to 512 columns stay with the registers, and up to 1024 with fewer than 16384 rows; so do calls that
// write the normalised tensor or read an fp32 gamma, by size (norm_rows_staged in rows_shape.cuh has the rule).
static bool norm_rows_swizzled(int64_t bpr, int64_t ld) { return bpr % 4 == 0 && ld % 64 == 0; }      // whole 64-element groups, a row a whole number of them from the next
constexpr int64_t kNormStagedSmem = 232448 - 2048;       // of a CTA for rows: less 1 KiB for the static part and 1 KiB for aligning
constexpr int kNormStagedMaxWarps = 32;
// acc + lo^2 + hi^2 for the two bf16 of a word, one rounding each
__device__ __forceinline__ float add_squares(uint32_t w, float acc) {
  asm("{ .reg .b16 l, h; mov.b32 {l, h}, %1; fma.rn.f32.bf16 %0, l, l, %0; fma.rn.f32.bf16 %0, h, h, %0; }" : "+f"(acc) : "r"(w));
  return acc;
}
__device__ __forceinline__ uint4 norm_lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
// Sums over the 32 lanes of kN values (a power of two, at most 8) at once, each in the order of a butterfly over lane
// distances 16, 8, 4, 2, 1: while there are several values a lane hands half of them to its partner and goes on with the other
// half.  Value j ends up in the lanes whose upper bits are j (total_of picks it).
template <int kN>
__device__ __forceinline__ float butterfly_sums(float (&v)[kN], int lane) {
  int o = 16;
#pragma unroll
  for (int n = kN / 2; n >= 1; n >>= 1, o >>= 1) {
    const bool upper = lane & o;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float other = __shfl_xor_sync(0xffffffffu, upper ? v[i] : v[i + n], o);
      v[i] = (upper ? v[i + n] : v[i]) + other;
    }
  }
#pragma unroll
  for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

template <typename TG, int kM, bool kWriteNorm>
__global__ void __launch_bounds__(kNormStagedMaxWarps * 32, 1)
rmsnorm_quantize_staged_kernel(const __grid_constant__ CUtensorMap map_x, const __nv_bfloat16* __restrict__ x, int rows, int blocks_per_row,
                             int64_t ld, const TG* __restrict__ gamma, float eps, uint2* __restrict__ codes,
                             float* __restrict__ amax_out, unsigned int* __restrict__ gmax,
                             unsigned int* __restrict__ records, void* __restrict__ norm_out, int swizzled, int bufs) {
  constexpr bool kProductBf16 = sizeof(TG) == 2;
  constexpr int kPow = kM <= 1 ? 1 : kM <= 2 ? 2 : kM <= 4 ? 4 : 8;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[2 * kNormStagedMaxWarps];
  __shared__ unsigned s_top[kNormStagedMaxWarps];
  __shared__ int s_failed[kNormStagedMaxWarps];             // by warp: gave up waiting for a row
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t row_bytes = (uint32_t)blocks_per_row * 32u, pitch = (row_bytes + 1023u) & ~1023u;
  const uint32_t s_gamma = base, mine = base + (kProductBf16 ? pitch : 0u) + (uint32_t)(warp * bufs) * pitch;
  uint64_t* my_full = full + 2 * warp;
  if (lane == 0) {
    for (int b = 0; b < bufs; ++b) mbar_init(&my_full[b], 1);
    s_failed[warp] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  grid_dependency_wait();
  __syncwarp();
  const int row_step = gridDim.x * warps;
  const int r_first = blockIdx.x * warps + warp;
  auto fetch = [&](int r, int b) {                        // lane 0
    mbar_expect_tx(&my_full[b], row_bytes);
    if (swizzled) tma_load_3d_addr(mine + b * pitch, &map_x, 0, 0, r, smem_u32(&my_full[b]));
    else          bulk_load_addr(mine + b * pitch, x + (int64_t)r * ld, row_bytes, smem_u32(&my_full[b]));
  };
  if (lane == 0) {
    for (int b = 0; b < bufs; ++b) if (r_first + b * row_step < rows) fetch(r_first + b * row_step, b);
  }
  // gamma as 16-byte pieces, piece c of each 128-byte group g at c ^ (g & 7); the barrier behind it stands after the first sum
  if constexpr (kProductBf16) {
    for (int p = threadIdx.x; p < 2 * blocks_per_row; p += blockDim.x) {
      const uint4 w = __ldg(reinterpret_cast<const uint4*>(gamma) + p);
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(s_gamma + (uint32_t)((p & ~7) | ((p ^ (p >> 3)) & 7)) * 16u), "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w) : "memory");
    }
  }
  bool gamma_there = !kProductBf16;
  // this lane's pieces of group of 32 blocks j: at these offsets + 1024 j
  const uint32_t group = (uint32_t)lane >> 2, swz0 = group * 128u + (((2u * (lane & 3u)) ^ (group & 7u)) << 4), swz1 = swz0 ^ 16u;
  const uint32_t x0 = swizzled ? swz0 : (uint32_t)lane * 32u, x1 = swizzled ? swz1 : (uint32_t)lane * 32u + 16u;
  const float n_cols = (float)(blocks_per_row * 16);
  const bool last_live = lane + 32 * (kM - 1) < blocks_per_row;     // of the lane's kM blocks only the last may be missing
  float running = 0.0f;
  volatile int* failed = &s_failed[warp];
  int b = 0;
  uint32_t parity = 0;
  bool gave_up = false;
  for (int r = r_first; r < rows; r += row_step) {
    const uint32_t row = mine + b * pitch;
    if (!__all_sync(0xffffffffu, mbar_wait(&my_full[b], parity, failed))) {
      gave_up = true;
      break;
    }
    float ss[kPow];
#pragma unroll
    for (int j = 0; j < kPow; ++j) {
      ss[j] = 0.0f;
      if (j < kM - 1 || (j == kM - 1 && last_live)) {
        const uint4 p = norm_lds128(row + x0 + 1024 * j), q = norm_lds128(row + x1 + 1024 * j);
        const uint32_t w[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) ss[j] = add_squares(w[i], ss[j]);
      }
    }
    const float sums = butterfly_sums<kPow>(ss, lane);
    float tot = 0.0f;
#pragma unroll
    for (int j = 0; j < kM; ++j) tot += __shfl_sync(0xffffffffu, sums, j * (32 / kPow));
    const float rs = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, n_cols), eps)));   // llama.py:23-24
    const f32x2 rs2 = pack2(rs, rs);
    if (!gamma_there) {                                    // uniform over the CTA: every warp comes here or to the same barrier below
      __syncthreads();
      gamma_there = true;
    }
    const int64_t row_blk = (int64_t)r * blocks_per_row + lane;
    uint2* row_codes = codes + row_blk;
    float* row_amax = amax_out + row_blk;
#pragma unroll
    for (int j = 0; j < kM; ++j) {
      if (j == kM - 1 && !last_live) break;
      RawBlock<__nv_bfloat16> raw;
      raw.a = norm_lds128(row + x0 + 1024 * j);
      raw.b = norm_lds128(row + x1 + 1024 * j);
      float v[16], y[16];
      raw.unpack(v);
      float a;
      if constexpr (kProductBf16) {
        const uint4 g0 = norm_lds128(s_gamma + swz0 + 1024 * j), g1 = norm_lds128(s_gamma + swz1 + 1024 * j);
        const uint32_t gw[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
        a = 0.0f;                                         // what a block of NaN has, as norm_block gives it
#pragma unroll
        for (int i = 0; i < 8; ++i) {                     // both roundings of the reference, see rmsnorm_quantize_kernel
          float n0, n1;
          split2(mul2(pack2(v[2 * i], v[2 * i + 1]), rs2), n0, n1);
          const __nv_bfloat162 n2 = __floats2bfloat162_rn(n0, n1);
          const __nv_bfloat162 p2 = __hmul2(n2, *reinterpret_cast<const __nv_bfloat162*>(&gw[i]));
          const uint32_t w = *reinterpret_cast<const uint32_t*>(&p2);
          y[2 * i] = bf16_lo(w);
          y[2 * i + 1] = bf16_hi(w);
          a = max3(a, fabsf(y[2 * i]), fabsf(y[2 * i + 1]));
        }
      } else {
        a = norm_block<__nv_bfloat16, TG>(v, rs, gamma + (lane + 32 * j) * 16, y);
      }
      uint32_t packed[2];
      quantize_rn<2>(y, block_scale_from_amax(a), packed);
      row_codes[32 * j] = make_uint2(packed[0], packed[1]);
      row_amax[32 * j] = a;
      running = fmaxf(running, a);
      if (kWriteNorm) {
        if (kProductBf16) {
          __nv_bfloat162 o[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = __floats2bfloat162_rn(y[2 * i], y[2 * i + 1]);   // exact: already bf16 values
          uint4* dst = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(norm_out) + (row_blk + 32 * j) * 16);
          dst[0] = reinterpret_cast<uint4*>(o)[0];
          dst[1] = reinterpret_cast<uint4*>(o)[1];
        } else {
          float4* dst = reinterpret_cast<float4*>(static_cast<float*>(norm_out) + (row_blk + 32 * j) * 16);
#pragma unroll
          for (int i = 0; i < 4; ++i) dst[i] = make_float4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]);
        }
      }
    }
    __syncwarp();                                          // every lane has read the row: its place takes another one
    const int next = r + bufs * row_step;
    if (lane == 0 && next < rows) fetch(next, b);
    if (++b == bufs) { b = 0; parity ^= 1u; }
  }
  if (!gamma_there) __syncthreads();
  if (gave_up && lane == 0) {
    *failed = 1;
    if (!records) gmax[1] = 1u;                            // error word: the scale pass publishes NaN as the unit
    // copies of this warp may still be in flight: give each a bounded chance to land before the CTA leaves
    for (int k = 0; k < bufs; ++k) {
      const uint64_t t0 = global_ns();
      while (!mbar_try(&my_full[b], parity) && global_ns() - t0 < kWaitLimitNs) {}
      if (++b == bufs) { b = 0; parity ^= 1u; }
    }
  }
  const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(running));       // >= 0: the bits order like the value
  if (!records) {
    if (lane == 0 && top > 0u) atomicMax(gmax, top);
    return;
  }
  if (lane == 0) s_top[warp] = top;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned m = 0u, bad = 0u;
    for (int w = 0; w < warps; ++w) { m = max(m, s_top[w]); bad |= (unsigned)s_failed[w]; }
    records[3 * blockIdx.x] = m;
    records[3 * blockIdx.x + 1] = 0u;
    records[3 * blockIdx.x + 2] = bad;
    if (blockIdx.x == 0) records[-1] = gridDim.x;
  }
}

constexpr int kNormSmallPasses = 2;
constexpr int kNormSmallThreads = 512;             // twice the rows per CTA of the streaming kernel: 16 rows of 4096 in one pass
constexpr int kNormSmallBlocks = 2;                // blocks per thread and row: rows of up to 8192 elements

template <typename TX, typename TG, int kBlocks, bool kWriteNorm>
__global__ void __launch_bounds__(kNormSmallThreads)
rmsnorm_quantize_small_kernel(const TX* __restrict__ x, int rows, int blocks_per_row, int64_t ld,
                              const TG* __restrict__ gamma, float eps, uint2* __restrict__ codes, int32_t sf_layout,
                              int tiles, int padded_words, uint8_t* __restrict__ scales, float* __restrict__ unit_out,
                              void* __restrict__ norm_out) {
  constexpr bool kProductBf16 = (sizeof(TX) == 2) && (sizeof(TG) == 2);
  __shared__ ClusterMaxSmem s_max;
  __shared__ float s_red[kNormSmallPasses][kNormSmallThreads / 32];
  __shared__ float s_rs[kNormSmallPasses][kNormSmallThreads / 32];
  grid_dependency_wait();
  const int bx = blockDim.x, by = blockDim.y;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int tid = ty * bx + tx;
  const int lane = tid & 31, warp = tid >> 5;
  const int seg = bx < 32 ? bx : 32;                 // lanes of one row inside a warp
  const int warps_per_row = bx >> 5;                 // 0 when a warp holds several rows
  const float n_cols = (float)(blocks_per_row * 16);
  const int ncta = (int)cluster_cta_count(), rank = (int)cluster_cta_rank();
  if (sf_layout == METIS_SF_MMA)
    zero_scale_padding(scales, rows, blocks_per_row, tiles, padded_words, rank * bx * by + tid, ncta * bx * by);

  // every row of this thread is on its way before the first one is worked on
  RawBlock<TX> raw[kNormSmallPasses][kBlocks];
#pragma unroll
  for (int p = 0; p < kNormSmallPasses; ++p) {
    const int r = (p * ncta + rank) * by + ty;
#pragma unroll
    for (int j = 0; j < kBlocks; ++j) {
      const int bc = tx + j * bx;
      if (r < rows && bc < blocks_per_row) raw[p][j].load(x + (int64_t)r * ld + (int64_t)bc * 16);
    }
  }
  // sums of squares of all passes, then one round through shared memory for all of them
  float ss[kNormSmallPasses];
#pragma unroll
  for (int p = 0; p < kNormSmallPasses; ++p) {
    const int r = (p * ncta + rank) * by + ty;
    ss[p] = 0.0f;
#pragma unroll
    for (int j = 0; j < kBlocks; ++j) {
      const int bc = tx + j * bx;
      if (r < rows && bc < blocks_per_row) {
        float v[16];
        raw[p][j].unpack(v);
#pragma unroll
        for (int i = 0; i < 16; ++i) ss[p] = __fmaf_rn(v[i], v[i], ss[p]);
      }
    }
    for (int o = seg >> 1; o > 0; o >>= 1) ss[p] += __shfl_xor_sync(0xffffffffu, ss[p], o);
    if (warps_per_row > 1 && lane == 0) s_red[p][warp] = ss[p];
  }
  float rs[kNormSmallPasses];
  if (warps_per_row > 1) {                             // uniform over the CTA
    __syncthreads();
    if (tx == 0) {
#pragma unroll
      for (int p = 0; p < kNormSmallPasses; ++p) {
        if ((p * ncta + rank) * by + ty >= rows) continue;
        float tot = 0.0f;
        for (int w = 0; w < warps_per_row; ++w) tot += s_red[p][ty * warps_per_row + w];
        s_rs[p][ty] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, n_cols), eps)));   // llama.py:23-24
      }
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < kNormSmallPasses; ++p) rs[p] = s_rs[p][ty];
  } else {
#pragma unroll
    for (int p = 0; p < kNormSmallPasses; ++p) rs[p] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss[p], n_cols), eps)));
  }

  float amax[kNormSmallPasses][kBlocks];
  float running = 0.0f;
#pragma unroll
  for (int p = 0; p < kNormSmallPasses; ++p) {
    const int r = (p * ncta + rank) * by + ty;
#pragma unroll
    for (int j = 0; j < kBlocks; ++j) {
      const int bc = tx + j * bx;
      amax[p][j] = 0.0f;
      if (!(r < rows && bc < blocks_per_row)) continue;
      float v[16], y[16];
      raw[p][j].unpack(v);
      const float a = norm_block<TX, TG>(v, rs[p], gamma + (int64_t)bc * 16, y);
      uint32_t packed[2];
      quantize_rn<2>(y, block_scale_from_amax(a), packed);
      const int64_t b = (int64_t)r * blocks_per_row + bc;
      codes[b] = make_uint2(packed[0], packed[1]);
      amax[p][j] = a;
      running = fmaxf(running, a);
      if (kWriteNorm) {
        if (kProductBf16) {
          __nv_bfloat162 o[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = __floats2bfloat162_rn(y[2 * i], y[2 * i + 1]);   // exact: already bf16 values
          uint4* dst = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(norm_out) + b * 16);
          dst[0] = reinterpret_cast<uint4*>(o)[0];
          dst[1] = reinterpret_cast<uint4*>(o)[1];
        } else {
          float4* dst = reinterpret_cast<float4*>(static_cast<float*>(norm_out) + b * 16);
#pragma unroll
          for (int i = 0; i < 4; ++i) dst[i] = make_float4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]);
        }
      }
    }
  }

  const float unit = __fdiv_rn(block_scale_from_amax(cluster_fmax(running, s_max)), 448.0f);   // quant.py:21-22
  if (rank == 0 && tid == 0) *unit_out = unit;
#pragma unroll
  for (int p = 0; p < kNormSmallPasses; ++p) {
    const int r = (p * ncta + rank) * by + ty;
#pragma unroll
    for (int j = 0; j < kBlocks; ++j) {
      const int bc = tx + j * bx;
      if (!(r < rows && bc < blocks_per_row)) continue;
      const float ratio = __fdiv_rn(block_scale_from_amax(amax[p][j]), unit);                 // quant.py:23
      const int64_t off = (sf_layout == METIS_SF_MMA) ? sf_mma_offset(r, bc, tiles) : (int64_t)r * blocks_per_row + bc;
      scales[off] = float_to_e4m3(ratio);
    }
  }
  cluster_leave();
}

// Launches the one-cluster kernel if [rows, cols] fits it; *taken says whether it did.
template <typename TX, typename TG>
static int32_t try_small(const TX* x, int64_t rows, int64_t cols, int64_t ld, const TG* gamma, float eps, uint8_t* codes,
                         int32_t sf_layout, uint8_t* scales, float* unit, void* norm_out, cudaStream_t st, bool* taken) {
  *taken = false;
  const int bpr = (int)(cols >> 4);
  int bx = 1;
  if (bpr >= 32) {
    bx = ((bpr + 31) / 32) * 32;
    if (bx > kNormThreads) bx = kNormThreads;
  } else {
    while (bx < bpr) bx <<= 1;
  }
  const int by = kNormSmallThreads / bx;
  const int per_thread = (bpr + bx - 1) / bx;
  const int64_t tiles = sf_tiles_per_row(cols);
  const int64_t padded_words = sf_layout == METIS_SF_MMA ? ceil_div(rows, 128) * 128 * tiles : 0;
  if (per_thread > kNormSmallBlocks || rows > (int64_t)kSmallCtas * kNormSmallPasses * by ||
      padded_words > kSmallMaxPaddedWords || !aligned16(scales))
    return METIS_OK;
  int64_t ctas = ceil_div(rows, by);
  const int64_t for_padding = ceil_div(padded_words / 4, kNormSmallThreads);     // CTAs without rows still clear padding
  if (ctas < for_padding) ctas = for_padding;
  if (ctas > kSmallCtas) ctas = kSmallCtas;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3((unsigned)bx, (unsigned)by);
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
#define METIS_NORM_SMALL(KB, WN)                                                                                       \
  METIS_CUDA_OK(cudaLaunchKernelEx(&cfg, rmsnorm_quantize_small_kernel<TX, TG, KB, WN>, x, (int)rows, bpr, ld, gamma, eps, c2, \
                                   sf_layout, (int)tiles, (int)padded_words, scales, unit, norm_out))
  if (per_thread <= 1) { if (norm_out) METIS_NORM_SMALL(1, true); else METIS_NORM_SMALL(1, false); }
  else                 { if (norm_out) METIS_NORM_SMALL(2, true); else METIS_NORM_SMALL(2, false); }
#undef METIS_NORM_SMALL
  *taken = true;
  return METIS_OK;
}

// CTAs of the CTA-per-row kernel: persistent, as many as are resident at once, so that all of them finish together
template <typename TX, typename TG, int kBlocks>
static int64_t norm_ctas(int64_t rows, int bx, bool with_norm, int sms) {
  const int by = kNormThreads / bx;
  const void* kern = with_norm ? reinterpret_cast<const void*>(rmsnorm_quantize_kernel<TX, TG, kBlocks, true>)
                               : reinterpret_cast<const void*>(rmsnorm_quantize_kernel<TX, TG, kBlocks, false>);
  const int64_t blocks = (int64_t)sms * resident_ctas(kern, bx * by, 0), need = ceil_div(rows, by);
  return blocks < need ? blocks : need;
}

// *records: in: where the per-CTA records may go (or nullptr); out: nullptr if the running maximum was used instead
template <typename TX, typename TG, int kBlocks>
static int32_t launch_norm(const TX* x, int64_t rows, int bpr, int bx, int64_t ld, const TG* gamma, float eps,
                           uint32_t* codes, const WorkspaceView& ws, unsigned int** records, void* norm_out, int sms, cudaStream_t st) {
  const int by = kNormThreads / bx;
  const int64_t blocks = norm_ctas<TX, TG, kBlocks>(rows, bx, norm_out != nullptr, sms);
  if (blocks > kMaxRecords) *records = nullptr;
  if (!*records) METIS_CUDA_OK(cudaMemsetAsync(ws.gmax, 0, 2 * sizeof(unsigned int), st));   // running maximum and error word
  const dim3 b((unsigned)bx, (unsigned)by);
  uint2* c2 = reinterpret_cast<uint2*>(codes);
  if (norm_out)
    METIS_CUDA_OK(launch_overlapped(kLaunchStream, rmsnorm_quantize_kernel<TX, TG, kBlocks, true>, dim3((unsigned)blocks), b, 0, st,
                                    x, (int)rows, bpr, ld, gamma, eps, c2, ws.amax, ws.gmax, *records, norm_out));
  else
    METIS_CUDA_OK(launch_overlapped(kLaunchStream, rmsnorm_quantize_kernel<TX, TG, kBlocks, false>, dim3((unsigned)blocks), b, 0, st,
                                    x, (int)rows, bpr, ld, gamma, eps, c2, ws.amax, ws.gmax, *records, norm_out));
  return METIS_OK;
}

// The warp-per-row kernels for [rows, 16 bpr] bf16, 32 <= bpr <= 256 (512 to 4096 columns): the row in registers,
template <typename TG, int kM>
static int32_t launch_norm_rows(const __nv_bfloat16* x, int64_t rows, int bpr, int64_t ld, const TG* gamma, float eps, uint32_t* codes,
                                const WorkspaceView& ws, unsigned int** records, void* norm_out, int sms, cudaStream_t st) {
  auto kern = norm_out ? rmsnorm_quantize_rows_kernel<TG, kM, true> : rmsnorm_quantize_rows_kernel<TG, kM, false>;
  int64_t blocks = (int64_t)sms * resident_ctas(reinterpret_cast<const void*>(kern), kNormRowThreads, 0);
  const int64_t need = ceil_div(rows, kNormRowThreads / 32);
  if (blocks > need) blocks = need;
  if (blocks > kMaxRecords) *records = nullptr;
  if (!*records) METIS_CUDA_OK(cudaMemsetAsync(ws.gmax, 0, 2 * sizeof(unsigned int), st));   // running maximum and error word
  METIS_CUDA_OK(launch_overlapped(kLaunchStream, kern, dim3((unsigned)blocks), dim3(kNormRowThreads), 0, st, x, (int)rows, bpr, ld, gamma, eps,
                                  reinterpret_cast<uint2*>(codes), ws.amax, ws.gmax, *records, norm_out));
  return METIS_OK;
}

// and in shared memory: a CTA per SM, as many warps as
// rows fit its shared memory (twice as many rows where there is room), no more than it takes to go round the same number of times.
template <typename TG, int kM>
static int32_t launch_norm_staged(const __nv_bfloat16* x, int64_t rows, int bpr, int64_t ld, const TG* gamma, float eps, uint32_t* codes,
                                const WorkspaceView& ws, unsigned int** records, void* norm_out, int sms, cudaStream_t st) {
  auto kern = norm_out ? rmsnorm_quantize_staged_kernel<TG, kM, true> : rmsnorm_quantize_staged_kernel<TG, kM, false>;
  const int64_t pitch = ceil_div((int64_t)bpr * 32, 1024) * 1024, room = kNormStagedSmem - (sizeof(TG) == 2 ? pitch : 0);
  int64_t warps = room / pitch;
  if (warps > kNormStagedMaxWarps) warps = kNormStagedMaxWarps;
  const int64_t rounds = ceil_div(rows, sms * warps);
  warps = ceil_div(rows, sms * rounds);
  const int64_t bufs = rounds > 1 && 2 * warps * pitch <= room ? 2 : 1;
  const int64_t blocks = ceil_div(rows, warps * rounds) < sms ? ceil_div(rows, warps * rounds) : sms;
  if (blocks > kMaxRecords) *records = nullptr;
  if (!*records) METIS_CUDA_OK(cudaMemsetAsync(ws.gmax, 0, 2 * sizeof(unsigned int), st));   // running maximum and error word
  const bool swizzled = norm_rows_swizzled(bpr, ld);
  CUtensorMap map = {};
  if (swizzled) {
    if (int32_t rc = make_row_map(&map, x, bpr / 4, rows, ld * 2, "x")) return rc;
  }
  const size_t smem = (size_t)((sizeof(TG) == 2 ? pitch : 0) + warps * bufs * pitch + 1024);
  METIS_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kNormStagedSmem + 1024)));
  METIS_CUDA_OK(launch_overlapped(kLaunchStream, kern, dim3((unsigned)blocks), dim3((unsigned)warps * 32), smem, st, map, x, (int)rows, bpr, ld, gamma, eps,
                                  reinterpret_cast<uint2*>(codes), ws.amax, ws.gmax, *records, norm_out, swizzled ? 1 : 0, (int)bufs));
  return METIS_OK;
}

template <typename TX, typename TG>
static int32_t dispatch_chunks(const TX* x, int64_t rows, int64_t cols, int64_t ld, const TG* gamma,
                               float eps, uint32_t* codes, const WorkspaceView& ws, unsigned int** records, void* norm_out,
                               int sms, cudaStream_t st) {
  const int bpr = (int)(cols >> 4);
  // threads along the row: whole warps, as many as the row has 32-block groups (hidden 1536 runs
  // with 96 threads per row and two rows per CTA instead of 128 with a quarter of them idle);
  // rows shorter than a warp take the next power of two
  int bx = 1;
  if (bpr >= 32) {
    bx = ((bpr + 31) / 32) * 32;
    if (bx > kNormThreads) bx = kNormThreads;
  } else {
    while (bx < bpr) bx <<= 1;
  }
  if constexpr (sizeof(TX) == 2) {
    // a warp per row from kNormRowsMinRows on, and where a CTA per row has more CTAs than there are records
    if (bpr >= 32 && bpr <= 256 &&
        (rows >= kNormRowsMinRows || (*records && norm_ctas<TX, TG, 1>(rows, bx, norm_out != nullptr, sms) > kMaxRecords))) {
      const bool staged = norm_rows_staged(rows, bpr, sizeof(TG) == 4, norm_out != nullptr, norm_rows_swizzled(bpr, ld));
      switch ((bpr + 31) / 32) {
        case 1: return launch_norm_rows<TG, 1>(x, rows, bpr, ld, gamma, eps, codes, ws, records, norm_out, sms, st);
#define METIS_NORM_ROWS(M)                                                                                                     \
  case M: return staged ? launch_norm_staged<TG, M>(x, rows, bpr, ld, gamma, eps, codes, ws, records, norm_out, sms, st)       \
                        : launch_norm_rows<TG, M>(x, rows, bpr, ld, gamma, eps, codes, ws, records, norm_out, sms, st)
        METIS_NORM_ROWS(2); METIS_NORM_ROWS(3); METIS_NORM_ROWS(4); METIS_NORM_ROWS(5);
        METIS_NORM_ROWS(6); METIS_NORM_ROWS(7); METIS_NORM_ROWS(8);
#undef METIS_NORM_ROWS
      }
    }
  }
  const int per_thread = (bpr + bx - 1) / bx;
  if (per_thread <= 1) return launch_norm<TX, TG, 1>(x, rows, bpr, bx, ld, gamma, eps, codes, ws, records, norm_out, sms, st);
  if (per_thread <= 2) return launch_norm<TX, TG, 2>(x, rows, bpr, bx, ld, gamma, eps, codes, ws, records, norm_out, sms, st);
  if (per_thread <= 3) return launch_norm<TX, TG, 3>(x, rows, bpr, bx, ld, gamma, eps, codes, ws, records, norm_out, sms, st);
  if (per_thread <= 5) return launch_norm<TX, TG, 5>(x, rows, bpr, bx, ld, gamma, eps, codes, ws, records, norm_out, sms, st);
  if (per_thread <= 8) return launch_norm<TX, TG, 8>(x, rows, bpr, bx, ld, gamma, eps, codes, ws, records, norm_out, sms, st);
  return fail(METIS_ERR_TOO_LARGE, "rmsnorm rows longer than %d elements are not supported", 8 * kNormThreads * 16);
}

// ---- RMSNorm with the column sums of its output (the mean-centred path) ------------------------------------
// The mean-centred quantizer (bitlinear.py:326-332) needs the column mean of the NORMALISED activation before
// it can quantize anything, so normalisation and quantization cannot share one pass.  This kernel is the first
// of the two: it reads x once, writes y = norm(x) * gamma (the reference's roundings, llama.py:23-31), the
// reciprocal RMS of every row (what a backward pass needs) and, per resident row slot, the sums of the y it
// produced for every column; col_mean_finish_kernel adds those in a fixed order.  The quantizer then reads y
// once for both orientations.  Same thread layout as rmsnorm_quantize_kernel: a thread keeps its column blocks
// for all the rows it sees, so the sums stay in registers.
template <typename TX, typename TG, int kBlocks>
__global__ void __launch_bounds__(kNormThreads)
rmsnorm_colsum_kernel(const TX* __restrict__ x, int rows, int blocks_per_row, int64_t ld, const TG* __restrict__ gamma,
                      float eps, void* __restrict__ norm_out, float* __restrict__ rstd_out, float* __restrict__ partial) {
  grid_dependency_wait();
  constexpr bool kProductBf16 = (sizeof(TX) == 2) && (sizeof(TG) == 2);
  __shared__ float s_red[kNormThreads / 32];
  __shared__ float s_rs[kNormThreads / 32];
  const int bx = blockDim.x, by = blockDim.y;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int tid = ty * bx + tx;
  const int lane = tid & 31, warp = tid >> 5;
  const int seg = bx < 32 ? bx : 32;
  const int warps_per_row = bx >> 5;
  const float n_cols = (float)(blocks_per_row * 16);
  float csum[kBlocks][16];
#pragma unroll
  for (int j = 0; j < kBlocks; ++j)
#pragma unroll
    for (int i = 0; i < 16; ++i) csum[j][i] = 0.0f;

  RawBlock<TX> raw[kBlocks];
  auto fetch = [&](int r_first) {
    const int r = r_first + ty;
#pragma unroll
    for (int j = 0; j < kBlocks; ++j) {
      const int bc = tx + j * bx;
      if (r < rows && bc < blocks_per_row) raw[j].load(x + (int64_t)r * ld + (int64_t)bc * 16);
    }
  };
  fetch(blockIdx.x * by);
  for (int r0 = blockIdx.x * by; r0 < rows; r0 += gridDim.x * by) {
    const int r = r0 + ty;
    const bool row_live = r < rows;
    float v[kBlocks][16];
    float ss = 0.0f;
#pragma unroll
    for (int j = 0; j < kBlocks; ++j) {
      const int bc = tx + j * bx;
      if (row_live && bc < blocks_per_row) {
        raw[j].unpack(v[j]);
#pragma unroll
        for (int i = 0; i < 16; ++i) ss = __fmaf_rn(v[j][i], v[j][i], ss);
      }
    }
    fetch(r0 + gridDim.x * by);
    for (int o = seg >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    float rs;
    if (warps_per_row > 1) {
      if (lane == 0) s_red[warp] = ss;
      __syncthreads();
      if (tx == 0) {
        float tot = 0.0f;
        for (int w = 0; w < warps_per_row; ++w) tot += s_red[ty * warps_per_row + w];
        s_rs[ty] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, n_cols), eps)));
      }
      __syncthreads();
      rs = s_rs[ty];
    } else {
      rs = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, n_cols), eps)));
    }
    if (row_live && tx == 0 && rstd_out) rstd_out[r] = rs;
#pragma unroll
    for (int j = 0; j < kBlocks; ++j) {
      const int bc = tx + j * bx;
      if (!(row_live && bc < blocks_per_row)) continue;
      float y[16];
      norm_block<TX, TG>(v[j], rs, gamma + (int64_t)bc * 16, y);
#pragma unroll
      for (int i = 0; i < 16; ++i) csum[j][i] += y[i];
      const int64_t b = (int64_t)r * blocks_per_row + bc;
      if (kProductBf16) {
        __nv_bfloat162 o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = __floats2bfloat162_rn(y[2 * i], y[2 * i + 1]);   // exact: already bf16 values
        uint4* dst = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(norm_out) + b * 16);
        dst[0] = reinterpret_cast<uint4*>(o)[0];
        dst[1] = reinterpret_cast<uint4*>(o)[1];
      } else {
        float4* dst = reinterpret_cast<float4*>(static_cast<float*>(norm_out) + b * 16);
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = make_float4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]);
      }
    }
  }
  // this row slot's sums: partial[slot][cols], slot = blockIdx.x * by + ty
  float* dst = partial + ((int64_t)blockIdx.x * by + ty) * (int64_t)blocks_per_row * 16;
#pragma unroll
  for (int j = 0; j < kBlocks; ++j) {
    const int bc = tx + j * bx;
    if (bc >= blocks_per_row) continue;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      reinterpret_cast<float4*>(dst + (int64_t)bc * 16)[i] = make_float4(csum[j][4 * i], csum[j][4 * i + 1], csum[j][4 * i + 2], csum[j][4 * i + 3]);
  }
}

// A CTA takes 32 columns: its eight warps fetch the row slots' sums into shared memory (coalesced, eight loads of a warp in
// flight), the first warp adds them up slot by slot: a fixed order.  Up to 32 slots it reads them itself, all at once.  A thread
// per column that walks all slots in global memory is a chain of loads: 13.4 us for 256 slots, 15.5 for 296 (hidden 4096), 5.5
// and 7.4 here (64 slots 4.5 -> 2.7); summing every eighth slot in a warp of its own takes 4.6 and 5.9 but changes the last bit
// of the means.
constexpr int kFinishSlots = 256;                          // slots per round: 32 KiB
constexpr int kFinishDirectSlots = 32, kFinishFewSlots = 16;
// A handful of slots (decode): a thread per column, all loads in flight.  Norm and mean, this / the kernel below, us: 1 x 4096
// 3.6 / 3.9, 8 x 3584 3.7 / 4.1, 16 x 1536 3.5 / 3.9, but 20 x 4096 4.7 / 4.3.
__global__ void __launch_bounds__(256)
rmsnorm_mean_finish_few_kernel(const float* __restrict__ partial, int slots, int64_t rows, int64_t cols, float* __restrict__ mean) {
  grid_dependency_wait();
  const int64_t c = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (c >= cols) return;
  float v[kFinishFewSlots], sum = 0.0f;
#pragma unroll
  for (int i = 0; i < kFinishFewSlots; ++i) v[i] = i < slots ? partial[i * cols + c] : 0.0f;
#pragma unroll
  for (int i = 0; i < kFinishFewSlots; ++i) if (i < slots) sum += v[i];
  mean[c] = __fdiv_rn(sum, (float)rows);
}
__global__ void __launch_bounds__(256)
rmsnorm_mean_finish_kernel(const float* __restrict__ partial, int64_t slots, int64_t rows, int64_t cols, float* __restrict__ mean) {
  __shared__ float s_part[kFinishSlots][32];
  grid_dependency_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t c = (int64_t)blockIdx.x * 32 + lane;
  float sum = 0.0f;
  if (slots <= kFinishDirectSlots) {
    if (warp != 0 || c >= cols) return;
    float v[kFinishDirectSlots];
#pragma unroll
    for (int i = 0; i < kFinishDirectSlots; ++i) v[i] = i < slots ? partial[i * cols + c] : 0.0f;
#pragma unroll
    for (int i = 0; i < kFinishDirectSlots; ++i) if (i < slots) sum += v[i];
    mean[c] = __fdiv_rn(sum, (float)rows);
    return;
  }
  for (int64_t base = 0; base < slots; base += kFinishSlots) {
    const int n = (int)(slots - base < kFinishSlots ? slots - base : kFinishSlots);
    if (base > 0) __syncthreads();                         // the previous round's sums have been read
    if (c < cols) {
      int i = warp;
#pragma unroll 8
      for (const int whole = warp + ((n - warp + 7) / 64) * 64; i < whole; i += 8) s_part[i][lane] = partial[(base + i) * cols + c];
      float v[8];                                          // the last ones not one by one
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = i + 8 * j < n ? partial[(base + i + 8 * j) * cols + c] : 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) if (i + 8 * j < n) s_part[i + 8 * j][lane] = v[j];
    }
    __syncthreads();
    if (warp == 0 && c < cols) {
#pragma unroll 8
      for (int i = 0; i < n; ++i) sum += s_part[i][lane];
    }
  }
  if (warp == 0 && c < cols) mean[c] = __fdiv_rn(sum, (float)rows);
}

struct NormShape { int bx, by, per_thread; };
static NormShape norm_shape(int bpr) {
  int bx = 1;
  if (bpr >= 32) {
    bx = ((bpr + 31) / 32) * 32;
    if (bx > kNormThreads) bx = kNormThreads;
  } else {
    while (bx < bpr) bx <<= 1;
  }
  return {bx, kNormThreads / bx, (bpr + bx - 1) / bx};
}
// row slots (CTAs x rows in flight per CTA) the kernel above runs with: two CTAs per SM
static int64_t colsum_ctas(int64_t rows, int by) {
  int64_t blocks = (int64_t)device_sm_count() * 2;
  const int64_t need = ceil_div(rows, by);
  return blocks > need ? need : blocks;
}

template <typename TX, typename TG>
static int32_t launch_colsum(const TX* x, int64_t rows, int64_t cols, int64_t ld, const TG* gamma, float eps, void* norm_out,
                             float* rstd, float* partial, cudaStream_t st) {
  const int bpr = (int)(cols >> 4);
  const NormShape sh = norm_shape(bpr);
  const dim3 g((unsigned)colsum_ctas(rows, sh.by)), b((unsigned)sh.bx, (unsigned)sh.by);
#define METIS_COLSUM(KB) METIS_CUDA_OK(launch_overlapped(kLaunchStream, rmsnorm_colsum_kernel<TX, TG, KB>, g, b, 0, st, x, (int)rows, bpr, ld, gamma, eps, norm_out, rstd, partial))
  if (sh.per_thread <= 1) METIS_COLSUM(1);
  else if (sh.per_thread <= 2) METIS_COLSUM(2);
  else if (sh.per_thread <= 3) METIS_COLSUM(3);
  else if (sh.per_thread <= 5) METIS_COLSUM(5);
  else return fail(METIS_ERR_TOO_LARGE, "rmsnorm rows longer than %d elements are not supported here", 5 * kNormThreads * 16);
#undef METIS_COLSUM
  return METIS_OK;
}

}  // namespace metis

using namespace metis;

extern "C" int32_t metis_rmsnorm_nvfp4_quantize(const void* x, int32_t x_dtype, int64_t rows, int64_t cols,
                                                int64_t ld, const void* gamma, int32_t gamma_dtype,
                                                float eps, int32_t sf_layout, uint8_t* codes,
                                                uint8_t* scales, float* unit, void* norm_out,
                                                void* workspace, int64_t workspace_bytes, void* stream) {
  if (!x || !gamma) return fail(METIS_ERR_BAD_ARGUMENT, "x or gamma is null");
  if ((x_dtype != METIS_DTYPE_BF16 && x_dtype != METIS_DTYPE_F32) ||
      (gamma_dtype != METIS_DTYPE_BF16 && gamma_dtype != METIS_DTYPE_F32))
    return fail(METIS_ERR_BAD_ARGUMENT, "unknown dtype");
  if (rows <= 0 || cols <= 0) return fail(METIS_ERR_BAD_SHAPE, "empty tensor [%lld, %lld]", (long long)rows, (long long)cols);
  if (ld < cols) return fail(METIS_ERR_BAD_ARGUMENT, "ld %lld < cols %lld", (long long)ld, (long long)cols);
  if (int32_t rc = check_quant_outputs(rows, cols, sf_layout, codes, scales, unit, workspace, workspace_bytes)) return rc;
  if (ld % 8 != 0 || !aligned16(x) || !aligned16(gamma) || (norm_out && !aligned16(norm_out)))
    return fail(METIS_ERR_BAD_ALIGNMENT, "x, gamma and norm_out must be 16-byte aligned and ld a multiple of 8");

  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int32_t rc;
  bool taken = false;
  if (x_dtype == METIS_DTYPE_BF16 && gamma_dtype == METIS_DTYPE_BF16)
    rc = try_small(static_cast<const __nv_bfloat16*>(x), rows, cols, ld, static_cast<const __nv_bfloat16*>(gamma), eps, codes, sf_layout, scales, unit, norm_out, st, &taken);
  else if (x_dtype == METIS_DTYPE_BF16)
    rc = try_small(static_cast<const __nv_bfloat16*>(x), rows, cols, ld, static_cast<const float*>(gamma), eps, codes, sf_layout, scales, unit, norm_out, st, &taken);
  else if (gamma_dtype == METIS_DTYPE_BF16)
    rc = try_small(static_cast<const float*>(x), rows, cols, ld, static_cast<const __nv_bfloat16*>(gamma), eps, codes, sf_layout, scales, unit, norm_out, st, &taken);
  else
    rc = try_small(static_cast<const float*>(x), rows, cols, ld, static_cast<const float*>(gamma), eps, codes, sf_layout, scales, unit, norm_out, st, &taken);
  if (rc || taken) return rc;
  const WorkspaceView ws = view_workspace(workspace);
  unsigned int* records = workspace_records(workspace, workspace_bytes, rows, cols);
  const int sms = device_sm_count();
  uint32_t* c32 = reinterpret_cast<uint32_t*>(codes);
  if (x_dtype == METIS_DTYPE_BF16 && gamma_dtype == METIS_DTYPE_BF16)
    rc = dispatch_chunks(static_cast<const __nv_bfloat16*>(x), rows, cols, ld, static_cast<const __nv_bfloat16*>(gamma), eps, c32, ws, &records, norm_out, sms, st);
  else if (x_dtype == METIS_DTYPE_BF16)
    rc = dispatch_chunks(static_cast<const __nv_bfloat16*>(x), rows, cols, ld, static_cast<const float*>(gamma), eps, c32, ws, &records, norm_out, sms, st);
  else if (gamma_dtype == METIS_DTYPE_BF16)
    rc = dispatch_chunks(static_cast<const float*>(x), rows, cols, ld, static_cast<const __nv_bfloat16*>(gamma), eps, c32, ws, &records, norm_out, sms, st);
  else
    rc = dispatch_chunks(static_cast<const float*>(x), rows, cols, ld, static_cast<const float*>(gamma), eps, c32, ws, &records, norm_out, sms, st);
  if (rc) return rc;
  METIS_CUDA_OK(cudaGetLastError());
  return launch_finalize(ws, rows, cols, sf_layout, scales, unit, st, nullptr, records, 0);
}


extern "C" int64_t metis_rmsnorm_mean_workspace_bytes(int64_t rows, int64_t cols) {
  if (rows <= 0 || cols <= 0 || cols % 16 != 0) return 0;
  const NormShape sh = norm_shape((int)(cols >> 4));
  return colsum_ctas(rows, sh.by) * sh.by * cols * (int64_t)sizeof(float);
}

extern "C" int32_t metis_rmsnorm_mean(const void* x, int32_t x_dtype, int64_t rows, int64_t cols, int64_t ld,
                                      const void* gamma, int32_t gamma_dtype, float eps, void* norm_out, float* rstd,
                                      float* mean, void* workspace, int64_t workspace_bytes, void* stream) {
  if (!x || !gamma || !norm_out || !mean || !workspace) return fail(METIS_ERR_BAD_ARGUMENT, "null pointer");
  if ((x_dtype != METIS_DTYPE_BF16 && x_dtype != METIS_DTYPE_F32) || (gamma_dtype != METIS_DTYPE_BF16 && gamma_dtype != METIS_DTYPE_F32))
    return fail(METIS_ERR_BAD_ARGUMENT, "unknown dtype");
  if (rows <= 0 || cols <= 0) return fail(METIS_ERR_BAD_SHAPE, "empty tensor [%lld, %lld]", (long long)rows, (long long)cols);
  if (cols % 16 != 0) return fail(METIS_ERR_BAD_SHAPE, "NVFP4 block shape (1, 16) does not divide tensor shape (%lld, %lld)", (long long)rows, (long long)cols);
  if (ld < cols || ld % 8 != 0 || !aligned16(x) || !aligned16(gamma) || !aligned16(norm_out) || !aligned16(workspace))
    return fail(METIS_ERR_BAD_ALIGNMENT, "x, gamma, norm_out and workspace must be 16-byte aligned and ld a multiple of 8");
  if (workspace_bytes < metis_rmsnorm_mean_workspace_bytes(rows, cols)) return fail(METIS_ERR_WORKSPACE, "workspace too small");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  float* partial = static_cast<float*>(workspace);
  int32_t rc;
  if (x_dtype == METIS_DTYPE_BF16 && gamma_dtype == METIS_DTYPE_BF16)
    rc = launch_colsum(static_cast<const __nv_bfloat16*>(x), rows, cols, ld, static_cast<const __nv_bfloat16*>(gamma), eps, norm_out, rstd, partial, st);
  else if (x_dtype == METIS_DTYPE_BF16)
    rc = launch_colsum(static_cast<const __nv_bfloat16*>(x), rows, cols, ld, static_cast<const float*>(gamma), eps, norm_out, rstd, partial, st);
  else if (gamma_dtype == METIS_DTYPE_BF16)
    rc = launch_colsum(static_cast<const float*>(x), rows, cols, ld, static_cast<const __nv_bfloat16*>(gamma), eps, norm_out, rstd, partial, st);
  else
    rc = launch_colsum(static_cast<const float*>(x), rows, cols, ld, static_cast<const float*>(gamma), eps, norm_out, rstd, partial, st);
  if (rc) return rc;
  const NormShape sh = norm_shape((int)(cols >> 4));
  const int64_t slots = colsum_ctas(rows, sh.by) * sh.by;
  if (slots <= kFinishFewSlots)
    METIS_CUDA_OK(launch_overlapped(kLaunchShort, rmsnorm_mean_finish_few_kernel, dim3((unsigned)ceil_div(cols, 256)), dim3(256), 0, st,
                                    (const float*)partial, (int)slots, rows, cols, mean));
  else
    METIS_CUDA_OK(launch_overlapped(kLaunchShort, rmsnorm_mean_finish_kernel, dim3((unsigned)ceil_div(cols, 32)), dim3(256), 0, st,
                                    (const float*)partial, slots, rows, cols, mean));
  return METIS_OK;
}

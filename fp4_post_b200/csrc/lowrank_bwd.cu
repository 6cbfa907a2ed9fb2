// Backward of the unquantized low-rank branch  y_u = (s . y_v) U^T  on the tensor core (sm_100a).
//
// The reference leaves these products to autograd: ulinear is a plain nn.Linear and the scaling by s a
// torch.mul (src/Metis/Metis/bitlinear.py:752-760, 872-879), so with G = grad_output [M, N] in bf16
//     d_ts = G U            [M, r]   contraction over N
//     dU   = G^T (s . y_v)  [N, r]   contraction over the tokens M
//     ds   = sum_m d_ts . y_v,   d_yv = d_ts . s
// Both products are skinny (r <= 256) and bound by the one read of G each needs.  One kernel serves
// both: a bf16 tcgen05 GEMM  D[Mg, Ng] = A [Mg, Kg] B [Ng, Kg]^T  whose operands may be stored either way
// round:
//     K-major   memory [rows = Mg or Ng, Kg contiguous]   (G for d_ts: Kg = N)
//     MN-major  memory [Kg rows, Mg or Ng contiguous]     (U [N, r] for d_ts; G and s . y_v for dU: Kg = M)
// so no operand is ever transposed in memory.  TMA boxes are 64 elements (128 bytes) wide, 128-byte
// swizzled; an MN-major operand tile is made of 64-element column boxes placed side by side (leading
// byte offset = one box), its 8-row groups 1024 bytes apart exactly like a K-major tile.
//
// One CTA per work item (128 rows of D, one K split): warp 0 TMA producer, warp 1 MMA issuer, warps 2-5
// epilogue (raw fp32 partial sums to scratch).  The small finish kernels add the splits in a fixed order
// and apply what autograd would: the bf16 roundings, the product with s, the reduction for ds.
// Every wait is bounded and reports through the status word.
#include "gemm_common.cuh"

namespace metis {

constexpr int kPanelThreads = 192;          // producer, issuer, 4 epilogue warps
constexpr int kPanelKStage = 64;            // elements of the contraction per pipeline stage
constexpr int kPanelABytes = 128 * 128;     // 128 rows of D x 64 bf16
constexpr int kPanelBoxBytes = 64 * 128;    // one MN-major box: 64 contraction rows x 64 elements

struct PanelParams {
  int64_t Mg, Ng, Kg;
  int32_t bn;                 // Ng rounded up to a multiple of 64: the MMA's N
  int32_t stages;
  int32_t splits, k_per_split;      // K stages per split
  float* partial;  int64_t ldp;     // [splits, Mg, ldp] fp32
  int32_t* status;
  // fused finish of d_ts = G U (one split only): d_yv, and per CTA the column sums of bf16(d_ts * y_v) for ds, then
  // those of d_yv for its mean: block_sums [tiles, 2, r]
  const __nv_bfloat16* yv;  int64_t ldyv;
  const void* s;  int32_t s_is_f32;
  __nv_bfloat16* d_yv;  int64_t ldd;
  float* block_sums;
  int32_t r;
};

static inline int panel_stage_bytes(int bn) { return kPanelABytes + bn * 128; }
static inline int panel_smem_bytes(int bn, int stages) { return stages * panel_stage_bytes(bn) + 1024 + 256 + 2 * 4 * 256 * 4; }

// Column sums of a 32 x 32 block held one row per lane: after five exchange-and-add steps lane l holds
// the sum of column l (31 shuffles instead of 160).
__device__ __forceinline__ float column_sums32(float (&v)[32], int lane) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int j = 0; j < off; ++j) {
      const float send = upper ? v[j] : v[j + off];
      const float keep = upper ? v[j + off] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  return v[0];
}

template <bool kAMn, bool kBMn, bool kDts>
__global__ void __launch_bounds__(kPanelThreads, 1)
bf16_panel_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const PanelParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int stage_bytes = kPanelABytes + p.bn * 128;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + p.stages * stage_bytes);
  uint64_t* full = bars;                       // [stages]
  uint64_t* empty = bars + p.stages;           // [stages]
  uint64_t* acc_full = bars + 2 * p.stages;
  uint64_t* drain = bars + 2 * p.stages + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * p.stages + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* s_colsum = reinterpret_cast<float*>(smem + p.stages * stage_bytes + 256);     // [2][4][256], fused finish only

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t tile_m = blockIdx.x / p.splits;
  const int split = (int)(blockIdx.x - tile_m * p.splits);
  const int k_iters_all = (int)((p.Kg + kPanelKStage - 1) / kPanelKStage);
  const int it0 = split * p.k_per_split;
  const int iters = (k_iters_all - it0 < p.k_per_split) ? k_iters_all - it0 : p.k_per_split;
  const uint32_t tmem_cols = p.bn <= 64 ? 64u : (p.bn <= 128 ? 128u : 256u);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1);
    mbar_init(drain, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_dependency_wait();

  if (warp == 0) {
    // ===== TMA producer =====
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t full_base = smem_u32(full);
    const int32_t m0 = (int32_t)(tile_m * 128);
    const int b_boxes = p.bn / 64;
    for (int it = 0; it < iters && ok; ++it) {
      ok = __all_sync(0xffffffffu, mbar_wait(&empty[stage], phase ^ 1u, abort_flag));
      if (!ok) {
        if (lane == 0) report(p.status, abort_flag, METIS_DEV_TIMEOUT_MMA);
        break;
      }
      const uint32_t sa = smem_base + stage * stage_bytes;
      const uint32_t sb = sa + kPanelABytes;
      const uint32_t bar = full_base + stage * 8;
      const int32_t k0 = (it0 + it) * kPanelKStage;
      if (elect_one()) {
        mbar_expect_tx_addr(bar, (uint32_t)stage_bytes);
        if (kAMn) {
          tma_load_2d_addr(sa, &map_a, m0, k0, bar);                       // [64 k rows, 64 columns of D's rows]
          tma_load_2d_addr(sa + kPanelBoxBytes, &map_a, m0 + 64, k0, bar);
        } else {
          tma_load_2d_addr(sa, &map_a, k0, m0, bar);                       // [128 rows, 64 k]
        }
        if (kBMn) {
          for (int h = 0; h < b_boxes; ++h) tma_load_2d_addr(sb + h * kPanelBoxBytes, &map_b, h * 64, k0, bar);
        } else {
          tma_load_2d_addr(sb, &map_b, k0, 0, bar);                        // [bn rows, 64 k]
        }
      }
      if (++stage == p.stages) { stage = 0; phase ^= 1u; }
    }
    grid_launch_dependents();
  } else if (warp == 1) {
    // ===== tensor-core issuer =====
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true, issued = false;
    const uint32_t empty_base = smem_u32(empty);
    // descriptor low words: address, and for an MN-major tile the distance between its 64-element
    // column boxes as the leading byte offset
    const uint32_t a_lead = kAMn ? (uint32_t)(kPanelBoxBytes >> 4) : 1u;
    const uint32_t b_lead = kBMn ? (uint32_t)(kPanelBoxBytes >> 4) : 1u;
    // one MMA takes 16 elements of the contraction: 32 bytes along a K-major row, 16 rows of an MN-major tile
    const uint32_t a_step = kAMn ? (16u * 128u) >> 4 : 2u;
    const uint32_t b_step = kBMn ? (16u * 128u) >> 4 : 2u;
    const uint32_t idesc = idesc_bf16(p.bn) | (kAMn ? (1u << 15) : 0u) | (kBMn ? (1u << 16) : 0u);
    for (int it = 0; it < iters; ++it) {
      ok = __all_sync(0xffffffffu, mbar_wait(&full[stage], phase, abort_flag));
      if (!ok) {
        if (lane == 0) report(p.status, abort_flag, METIS_DEV_TIMEOUT_TMA);
        break;
      }
      tc_fence_after();
      const uint32_t sa = smem_u32(smem) + stage * stage_bytes;
      const uint32_t a_lo = ((sa & 0x3FFFFu) >> 4) | (a_lead << 16);
      const uint32_t b_lo = (((sa + kPanelABytes) & 0x3FFFFu) >> 4) | (b_lead << 16);
      if (elect_one()) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          tc_mma_bf16(tmem_base, a_lo + a_step * j, b_lo + b_step * j, kOperandDescHi, idesc, (it > 0 || j > 0) ? 1u : 0u);
        tc_commit_addr(empty_base + stage * 8);
        if (it == iters - 1) tc_commit(acc_full);
      }
      issued = true;
      if (++stage == p.stages) { stage = 0; phase ^= 1u; }
    }
    if (!ok && issued && elect_one()) {
      tc_commit(drain);
      const uint64_t t0 = global_ns();
      while (!mbar_try(drain, 0) && global_ns() - t0 < kWaitLimitNs) {}
    }
    __syncwarp();
  } else {
    // ===== epilogue: warps 2..5 own tensor-memory lanes 32*(warp%4) .. +31 =====
    const int q = warp & 3;
    const int64_t row = tile_m * 128 + q * 32 + lane;
    if (iters > 0) {
      if (!mbar_wait(acc_full, 0, abort_flag)) {
        if (lane == 0) report(p.status, abort_flag, METIS_DEV_TIMEOUT_MMA);
      } else {
        tc_fence_after();
        const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16);
        if constexpr (kDts) {
          // autograd's bf16 steps on this CTA's 128 rows of d_ts, straight from the accumulator
          const bool live = row < p.Mg;
          for (int ch = 0; ch * 32 < p.r; ++ch) {
            uint32_t acc[32];
            tc_load32(t_row + ch * 32, acc);
            uint32_t yw[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) yw[i] = 0u;
            if (live) {
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                if (ch * 32 + 8 * i < p.r) {
                  const uint4 w = __ldg(reinterpret_cast<const uint4*>(p.yv + row * p.ldyv + ch * 32) + i);
                  yw[4 * i] = w.x; yw[4 * i + 1] = w.y; yw[4 * i + 2] = w.z; yw[4 * i + 3] = w.w;
                }
              }
            }
            tc_wait_ld(acc);
            float prod[32], dyv[32];
            uint32_t ow[16];
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const int c = ch * 32 + i;
              float s0 = 0.0f, s1 = 0.0f;
              if (c < p.r) {
                if (p.s_is_f32) { s0 = static_cast<const float*>(p.s)[c]; s1 = static_cast<const float*>(p.s)[c + 1]; }
                else { const uint32_t sw = *reinterpret_cast<const uint32_t*>(static_cast<const __nv_bfloat16*>(p.s) + c); s0 = bf16_lo(sw); s1 = bf16_hi(sw); }
              }
              const __nv_bfloat162 s2 = __floats2bfloat162_rn(s0, s1);                             // s.to(bf16)
              const __nv_bfloat162 d2 = __floats2bfloat162_rn(__uint_as_float(acc[i]), __uint_as_float(acc[i + 1]));   // the product's bf16 output
              const __nv_bfloat162 o2 = __hmul2(d2, s2);                                             // d_ts * s, one rounding
              const __nv_bfloat162 p2 = __hmul2(d2, *reinterpret_cast<const __nv_bfloat162*>(&yw[i >> 1]));   // d_ts * y_v
              ow[i >> 1] = *reinterpret_cast<const uint32_t*>(&o2);
              const uint32_t pw = *reinterpret_cast<const uint32_t*>(&p2);
              prod[i] = live ? bf16_lo(pw) : 0.0f;
              prod[i + 1] = live ? bf16_hi(pw) : 0.0f;
              dyv[i] = live ? bf16_lo(ow[i >> 1]) : 0.0f;
              dyv[i + 1] = live ? bf16_hi(ow[i >> 1]) : 0.0f;
            }
            if (live) {
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (ch * 32 + 8 * i < p.r)
                  reinterpret_cast<uint4*>(p.d_yv + row * p.ldd + ch * 32)[i] = make_uint4(ow[4 * i], ow[4 * i + 1], ow[4 * i + 2], ow[4 * i + 3]);
            }
            s_colsum[q * 256 + ch * 32 + lane] = column_sums32(prod, lane);
            s_colsum[1024 + q * 256 + ch * 32 + lane] = column_sums32(dyv, lane);
          }
        } else {
          float* dst = p.partial + ((int64_t)split * p.Mg + row) * p.ldp;
          for (int ch = 0; ch < p.bn / 32; ++ch) {
            uint32_t r[32];
            tc_load32(t_row + ch * 32, r);
            tc_wait_ld(r);
            if (row < p.Mg && ch * 32 < p.ldp) {
#pragma unroll
              for (int i = 0; i < 8; ++i)
                reinterpret_cast<float4*>(dst + ch * 32)[i] =
                    make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
            }
          }
        }
        tc_fence_before();
      }
    } else if (row < p.Mg) {
      // a split without iterations contributes zeros
      float* dst = p.partial + ((int64_t)split * p.Mg + row) * p.ldp;
      for (int64_t c = 0; c < p.ldp; ++c) dst[c] = 0.0f;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
  if constexpr (kDts) {
    // this CTA's column sums, its four 32-row groups in a fixed order (lowrank_ds_kernel adds the CTAs')
    for (int c = threadIdx.x; c < p.r; c += kPanelThreads) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float* part = s_colsum + 1024 * k + c;
        p.block_sums[((int64_t)blockIdx.x * 2 + k) * p.r + c] = (part[0] + part[256]) + (part[512] + part[768]);
      }
    }
  }
}

// ---- finish kernels -------------------------------------------------------------------------------------------

// d_ts = bf16(sum over splits); d_yv = bf16(d_ts * bf16(s)); per-CTA column sums of bf16(d_ts * y_v) and of d_yv
// go to block_sums [gridDim.x, 2, r], which lowrank_ds_kernel adds into ds and the column mean of d_yv.
// A thread takes four columns of a row and has the partial sums of all splits in flight before it adds them; a CTA
// takes 512 / r rows at a time and the grid as many CTAs as there are such groups (up to kDtsFinishCtas).  Bound by
// the read of the partial sums (1120 x 128, 7 splits, with the product and the sums behind it: 13 us; 58 with a column
// per thread and one load in flight).  128 threads of up to 64 registers, because the CTAs run beside a weight-gradient
// product whose own CTA leaves 22 K registers of an SM: larger ones wait for that product to end.
constexpr int kFinishThreads = 128;
constexpr int kPanelMaxSplits = 16;
// v += the partial sums at src of all splits, in split order, eight loads in flight
__device__ __forceinline__ void add_splits(const float* __restrict__ src, int splits, int64_t split_pitch, float (&v)[4]) {
  for (int sp0 = 0; sp0 < splits; sp0 += 8) {
    float4 part[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (sp0 + i < splits) part[i] = *reinterpret_cast<const float4*>(src + (int64_t)(sp0 + i) * split_pitch);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (sp0 + i < splits) { v[0] += part[i].x; v[1] += part[i].y; v[2] += part[i].z; v[3] += part[i].w; }
  }
}
__global__ void __launch_bounds__(kFinishThreads, 7)
lowrank_dts_finish_kernel(const float* __restrict__ partial, int splits, int64_t M, int r, int64_t ldp,
                          const __nv_bfloat16* __restrict__ yv, int64_t ldyv, const void* __restrict__ s, int s_is_f32,
                          __nv_bfloat16* __restrict__ d_yv, int64_t ldd, float* __restrict__ block_sums) {
  grid_dependency_wait();
  const int groups = r >> 2, lanes = kFinishThreads / groups;      // threads of a row, rows at a time
  const int cg = threadIdx.x % groups, ry = threadIdx.x / groups;
  const int c = cg * 4;
  __shared__ float4 s_sum[2][kFinishThreads];                      // [lanes][groups]
  float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f}, acc_o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  if (ry < lanes) {
    float sc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      sc[j] = s_is_f32 ? __bfloat162float(__float2bfloat16_rn(static_cast<const float*>(s)[c + j]))
                       : __bfloat162float(static_cast<const __nv_bfloat16*>(s)[c + j]);
    for (int64_t row = (int64_t)blockIdx.x * lanes + ry; row < M; row += (int64_t)gridDim.x * lanes) {
      const float* src = partial + row * ldp + c;
      const uint2 yw = *reinterpret_cast<const uint2*>(yv + row * ldyv + c);
      float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      add_splits(src, splits, M * ldp, v);
      const float y[4] = {bf16_lo(yw.x), bf16_hi(yw.x), bf16_lo(yw.y), bf16_hi(yw.y)};
      __nv_bfloat16 o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float dts = __bfloat162float(__float2bfloat16_rn(v[j]));                   // the product's bf16 output
        o[j] = __float2bfloat16_rn(dts * sc[j]);
        acc[j] += __bfloat162float(__float2bfloat16_rn(dts * y[j]));
        acc_o[j] += __bfloat162float(o[j]);
      }
      *reinterpret_cast<uint2*>(d_yv + row * ldd + c) = *reinterpret_cast<const uint2*>(o);
    }
    s_sum[0][ry * groups + cg] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    s_sum[1][ry * groups + cg] = make_float4(acc_o[0], acc_o[1], acc_o[2], acc_o[3]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * groups; i += kFinishThreads) {
    const int k = i >= groups, col = i - k * groups;
    float4 t = s_sum[k][col];
    for (int l = 1; l < lanes; ++l) {
      const float4 u = s_sum[k][l * groups + col];
      t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
    }
    *reinterpret_cast<float4*>(block_sums + ((int64_t)blockIdx.x * 2 + k) * r + 4 * col) = t;
  }
}

// ds[c] (blockIdx.y 0) and the column mean of d_yv (1): sums of block_sums[b][y][c] over the blocks, in a fixed order: a
// warp takes 32 columns and every eighth block, the eight warps' sums are added in order.  A launch of its own: the last
// CTA of the kernel that writes block_sums could add them too, but the fence and the ticket that takes cost that
// kernel 12-17 us.  The mean replaces a pass over d_yv of two launches (8 us of the step's critical chain).
template <typename TS>
__global__ void __launch_bounds__(256)
lowrank_ds_kernel(const float* __restrict__ block_sums, int blocks, int r, float rows, TS* __restrict__ ds, float* __restrict__ mean) {
  grid_dependency_wait();
  __shared__ float s_part[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane, y = blockIdx.y;
  float acc = 0.0f;
  if (c < r) {
#pragma unroll 16
    for (int b = warp; b < blocks; b += 8) acc += block_sums[((int64_t)b * 2 + y) * r + c];
  }
  s_part[warp][lane] = acc;
  __syncthreads();
  if (warp == 0 && c < r) {
    float total = s_part[0][lane];
#pragma unroll
    for (int w = 1; w < 8; ++w) total += s_part[w][lane];
    if (y == 1) mean[c] = __fdiv_rn(total, rows);
    else if constexpr (sizeof(TS) == 2) ds[c] = __float2bfloat16_rn(total);
    else ds[c] = total;
  }
}

// Sum over the splits, four columns per thread (`vec`: they can be stored at once).  The block is (threads of a row, rows at a
// time): the two divisions by the width that a flat block needs cost 0.1-0.2 us of a small call (1000 x 1040 x 8 7.1 -> 6.9).
template <typename TU>
__global__ void __launch_bounds__(kFinishThreads, 7)
lowrank_du_finish_kernel(const float* __restrict__ partial, int splits, int64_t N, int r, int64_t ldp,
                         TU* __restrict__ grad_u, int64_t ldu, bool vec) {
  grid_dependency_wait();
  const uint32_t lanes = blockDim.y, ry = threadIdx.y;
  const int c = (int)threadIdx.x * 4;
  for (int64_t n = (int64_t)blockIdx.x * lanes + ry; n < N; n += (int64_t)gridDim.x * lanes) {
    const float* src = partial + n * ldp + c;                     // the partial sums fill whole 64-column panels
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    add_splits(src, splits, N * ldp, v);
    TU* dst = grad_u + n * ldu + c;
    if constexpr (sizeof(TU) == 2) {
      __nv_bfloat162 o[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
      if (vec) {
        *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(o);
      } else {
        for (int j = 0; j < 4 && c + j < r; ++j) dst[j] = reinterpret_cast<const __nv_bfloat16*>(o)[j];
      }
    } else {
      if (vec) {
        *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
        for (int j = 0; j < 4 && c + j < r; ++j) dst[j] = v[j];
      }
    }
  }
}

// ---- host side ----------------------------------------------------------------------------------------------

struct PanelPlan {
  int bn, stages, splits, k_per_split;
  int64_t ldp, tiles_m, partial_bytes;
};

static PanelPlan plan_panel(int64_t Mg, int64_t Ng, int64_t Kg) {
  PanelPlan pl;
  pl.bn = (int)(ceil_div(Ng, 64) * 64);
  pl.stages = pl.bn <= 128 ? 6 : 4;
  pl.tiles_m = ceil_div(Mg, 128);
  const int64_t k_iters = ceil_div(Kg, kPanelKStage);
  // enough work items to fill the SMs once, never fewer than 8 K stages per split
  int64_t s = device_sm_count() / pl.tiles_m;
  if (s > k_iters / 8) s = k_iters / 8;
  if (s > kPanelMaxSplits) s = kPanelMaxSplits;
  if (s < 1) s = 1;
  pl.k_per_split = (int)ceil_div(k_iters, s);
  pl.splits = (int)ceil_div(k_iters, pl.k_per_split);
  pl.ldp = pl.bn;
  pl.partial_bytes = (int64_t)pl.splits * Mg * pl.ldp * (int64_t)sizeof(float);
  return pl;
}

// D partial sums [splits, Mg, ldp]; a: [Mg, Kg] (K-major) or [Kg, Mg] (MN-major), b likewise with Ng
static int32_t launch_panel(const void* a, bool a_mn, int64_t lda, const void* b, bool b_mn, int64_t ldb, int64_t Mg, int64_t Ng,
                            int64_t Kg, const PanelPlan& pl, float* partial, int32_t* status, cudaStream_t st,
                            const PanelParams* dts = nullptr) {
  CUtensorMap ma, mb;
  const CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  if (a_mn) { if (int32_t rc = make_map(&ma, dt, 2, a, Mg, Kg, lda * 2, 64, kPanelKStage, "A (MN-major)")) return rc; }
  else      { if (int32_t rc = make_map(&ma, dt, 2, a, Kg, Mg, lda * 2, 64, 128, "A (K-major)")) return rc; }
  if (b_mn) { if (int32_t rc = make_map(&mb, dt, 2, b, Ng, Kg, ldb * 2, 64, kPanelKStage, "B (MN-major)")) return rc; }
  else      { if (int32_t rc = make_map(&mb, dt, 2, b, Kg, Ng, ldb * 2, 64, pl.bn, "B (K-major)")) return rc; }
  PanelParams p = {};
  if (dts) p = *dts;
  p.Mg = Mg; p.Ng = Ng; p.Kg = Kg; p.bn = pl.bn; p.stages = pl.stages; p.splits = pl.splits; p.k_per_split = pl.k_per_split;
  p.partial = partial; p.ldp = pl.ldp; p.status = status;
  const int smem = panel_smem_bytes(pl.bn, pl.stages);
  const dim3 grid((unsigned)(pl.tiles_m * pl.splits)), block(kPanelThreads);
#define METIS_LAUNCH_PANEL(AMN, BMN)                                                                         \
  do {                                                                                                       \
    auto kern = bf16_panel_gemm_kernel<AMN, BMN, false>;                                                     \
    METIS_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));            \
    METIS_CUDA_OK(launch_overlapped(kLaunchGemm, kern, grid, block, (size_t)smem, st, ma, mb, p));           \
  } while (0)
  if (dts) {                                   // d_ts = G U with the fused finish: K-major G, U read as it lies
    auto kern = bf16_panel_gemm_kernel<false, true, true>;
    METIS_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    METIS_CUDA_OK(launch_overlapped(kLaunchGemm, kern, grid, block, (size_t)smem, st, ma, mb, p));
    return METIS_OK;
  }
  if (a_mn) { if (b_mn) METIS_LAUNCH_PANEL(true, true); else METIS_LAUNCH_PANEL(true, false); }
  else      { if (b_mn) METIS_LAUNCH_PANEL(false, true); else METIS_LAUNCH_PANEL(false, false); }
#undef METIS_LAUNCH_PANEL
  return METIS_OK;
}

template <typename TU>
static int32_t launch_sum(const float* partial, const PanelPlan& pl, int64_t rows, int64_t r, TU* out, int64_t ld, cudaStream_t st) {
  const int64_t groups = ceil_div(r, 4), lanes = kFinishThreads / groups;          // threads of a row, rows at a time
  int64_t blocks = ceil_div(rows, lanes);
  if (blocks > (int64_t)device_sm_count() * 8) blocks = (int64_t)device_sm_count() * 8;
  const bool vec = r % 4 == 0 && ld % 4 == 0 && aligned16(out);
  METIS_CUDA_OK(launch_overlapped(kLaunchShort, lowrank_du_finish_kernel<TU>, dim3((unsigned)blocks), dim3((unsigned)groups, (unsigned)lanes), 0, st,
                                  partial, pl.splits, rows, (int)r, pl.ldp, out, ld, vec));
  return METIS_OK;
}

static int32_t check_bf16_matrix(const void* p, int64_t ld, int64_t cols, const char* what) {
  if (!p) return fail(METIS_ERR_BAD_ARGUMENT, "%s is null", what);
  if (!aligned16(p) || ld < cols || ld % 8 != 0) return fail(METIS_ERR_BAD_ALIGNMENT, "%s must be 16-byte aligned with a leading dimension that is a multiple of 8", what);
  return METIS_OK;
}

constexpr int kDtsFinishCtas = 256;
// per-CTA column sums: the finish kernel's CTAs, or one per 128 rows when the finish is fused
static int64_t dts_tail_bytes(int64_t M, int64_t r) {
  const int64_t ctas = ceil_div(M, 128) > kDtsFinishCtas ? ceil_div(M, 128) : kDtsFinishCtas;
  return 2 * ctas * r * (int64_t)sizeof(float);
}

}  // namespace metis

using namespace metis;

extern "C" int64_t metis_bf16_panel_gemm_workspace_bytes(int64_t Mg, int64_t Ng, int64_t Kg) {
  if (Mg <= 0 || Ng <= 0 || Kg <= 0) return 0;
  return plan_panel(Mg, Ng, Kg).partial_bytes;
}

extern "C" int32_t metis_bf16_panel_gemm(const void* a, int32_t a_mn_major, int64_t lda, const void* b, int32_t b_mn_major, int64_t ldb,
                                         int64_t Mg, int64_t Ng, int64_t Kg, float* d, int64_t ldd, void* workspace,
                                         int64_t workspace_bytes, int32_t* status, void* stream) {
  if (Mg <= 0 || Ng <= 0 || Kg <= 0) return fail(METIS_ERR_BAD_SHAPE, "empty product %lld x %lld x %lld", (long long)Mg, (long long)Ng, (long long)Kg);
  if (Ng > 256) return fail(METIS_ERR_BAD_SHAPE, "Ng = %lld: the panel product takes up to 256 columns", (long long)Ng);
  if (int32_t rc = check_bf16_matrix(a, lda, a_mn_major ? Mg : Kg, "a")) return rc;
  if (int32_t rc = check_bf16_matrix(b, ldb, b_mn_major ? Ng : Kg, "b")) return rc;
  if (!d || !workspace || ldd < Ng) return fail(METIS_ERR_BAD_ARGUMENT, "null pointer or ldd < Ng");
  if (!aligned16(workspace) || workspace_bytes < metis_bf16_panel_gemm_workspace_bytes(Mg, Ng, Kg)) return fail(METIS_ERR_WORKSPACE, "workspace too small or misaligned");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const PanelPlan pl = plan_panel(Mg, Ng, Kg);
  float* partial = static_cast<float*>(workspace);
  if (int32_t rc = launch_panel(a, a_mn_major != 0, lda, b, b_mn_major != 0, ldb, Mg, Ng, Kg, pl, partial, status, st)) return rc;
  return launch_sum(partial, pl, Mg, Ng, d, ldd, st);
}

extern "C" int64_t metis_lowrank_dts_workspace_bytes(int64_t M, int64_t N, int64_t r) {
  if (M <= 0 || N <= 0 || r <= 0) return 0;
  return plan_panel(M, r, N).partial_bytes + dts_tail_bytes(M, r);
}

extern "C" int32_t metis_lowrank_dts_mean(const void* g, int64_t ldg, int64_t M, int64_t N, const void* u, int64_t ldu, int64_t r,
                                          const void* yv, int64_t ldyv, const void* s, int32_t s_dtype, void* d_yv, int64_t ldd,
                                          void* ds, int32_t ds_dtype, float* d_yv_mean, void* workspace, int64_t workspace_bytes,
                                          int32_t* status, void* stream) {
  if (ds_dtype != METIS_DTYPE_BF16 && ds_dtype != METIS_DTYPE_F32) return fail(METIS_ERR_BAD_ARGUMENT, "unknown ds_dtype %d", ds_dtype);
  if (M <= 0 || N <= 0 || r <= 0) return fail(METIS_ERR_BAD_SHAPE, "empty product %lld x %lld x %lld", (long long)M, (long long)N, (long long)r);
  if (r > 256 || r % 8 != 0 || N % 8 != 0) return fail(METIS_ERR_BAD_SHAPE, "rank %lld must be a multiple of 8 up to 256 and N = %lld a multiple of 8", (long long)r, (long long)N);
  if (int32_t rc = check_bf16_matrix(g, ldg, N, "g")) return rc;
  if (int32_t rc = check_bf16_matrix(u, ldu, r, "u")) return rc;
  if (int32_t rc = check_bf16_matrix(yv, ldyv, r, "yv")) return rc;
  if (int32_t rc = check_bf16_matrix(d_yv, ldd, r, "d_yv")) return rc;
  if (!s || !ds || !workspace) return fail(METIS_ERR_BAD_ARGUMENT, "null pointer");
  if (s_dtype != METIS_DTYPE_BF16 && s_dtype != METIS_DTYPE_F32) return fail(METIS_ERR_BAD_ARGUMENT, "unknown s_dtype %d", s_dtype);
  if (!aligned16(workspace) || workspace_bytes < metis_lowrank_dts_workspace_bytes(M, N, r)) return fail(METIS_ERR_WORKSPACE, "workspace too small or misaligned");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const PanelPlan pl = plan_panel(M, r, N);
  float* partial = static_cast<float*>(workspace);
  float* block_sums = reinterpret_cast<float*>(static_cast<char*>(workspace) + pl.partial_bytes);
  int64_t blocks;
  // d_ts = G U: G [M, N] is K-major (contraction over its columns), U [N, r] holds the contraction in its rows
  if (pl.splits == 1) {
    // one split (many tokens): d_yv and ds come straight from the accumulator, no partial sums in memory
    PanelParams f = {};
    f.yv = static_cast<const __nv_bfloat16*>(yv); f.ldyv = ldyv; f.s = s; f.s_is_f32 = (s_dtype == METIS_DTYPE_F32);
    f.d_yv = static_cast<__nv_bfloat16*>(d_yv); f.ldd = ldd; f.block_sums = block_sums; f.r = (int32_t)r;
    if (int32_t rc = launch_panel(g, false, ldg, u, true, ldu, M, r, N, pl, partial, status, st, &f)) return rc;
    blocks = pl.tiles_m;
  } else {
    if (int32_t rc = launch_panel(g, false, ldg, u, true, ldu, M, r, N, pl, partial, status, st)) return rc;
    blocks = ceil_div(M, kFinishThreads / (r / 4));
    if (blocks > kDtsFinishCtas) blocks = kDtsFinishCtas;
    METIS_CUDA_OK(launch_overlapped(kLaunchShort, lowrank_dts_finish_kernel, dim3((unsigned)blocks), dim3(kFinishThreads), 0, st,
                                    (const float*)partial, pl.splits, M, (int)r, pl.ldp, static_cast<const __nv_bfloat16*>(yv), ldyv, s,
                                    (int)(s_dtype == METIS_DTYPE_F32), static_cast<__nv_bfloat16*>(d_yv), ldd, block_sums));
  }
  const dim3 grid((unsigned)ceil_div(r, 32), d_yv_mean ? 2 : 1);
  if (ds_dtype == METIS_DTYPE_BF16)
    METIS_CUDA_OK(launch_overlapped(kLaunchShort, lowrank_ds_kernel<__nv_bfloat16>, grid, dim3(256), 0, st, (const float*)block_sums,
                                    (int)blocks, (int)r, (float)M, static_cast<__nv_bfloat16*>(ds), d_yv_mean));
  else
    METIS_CUDA_OK(launch_overlapped(kLaunchShort, lowrank_ds_kernel<float>, grid, dim3(256), 0, st, (const float*)block_sums,
                                    (int)blocks, (int)r, (float)M, static_cast<float*>(ds), d_yv_mean));
  return METIS_OK;
}

extern "C" int32_t metis_lowrank_dts(const void* g, int64_t ldg, int64_t M, int64_t N, const void* u, int64_t ldu, int64_t r,
                                     const void* yv, int64_t ldyv, const void* s, int32_t s_dtype, void* d_yv, int64_t ldd,
                                     float* ds, void* workspace, int64_t workspace_bytes, int32_t* status, void* stream) {
  return metis_lowrank_dts_mean(g, ldg, M, N, u, ldu, r, yv, ldyv, s, s_dtype, d_yv, ldd, ds, METIS_DTYPE_F32, nullptr, workspace,
                                workspace_bytes, status, stream);
}

extern "C" int64_t metis_lowrank_du_workspace_bytes(int64_t M, int64_t N, int64_t r) {
  if (M <= 0 || N <= 0 || r <= 0) return 0;
  return plan_panel(N, r, M).partial_bytes;
}

extern "C" int32_t metis_lowrank_du(const void* g, int64_t ldg, int64_t M, int64_t N, const void* ts, int64_t ldts, int64_t r,
                                    void* grad_u, int32_t u_dtype, int64_t ldgu, void* workspace, int64_t workspace_bytes,
                                    int32_t* status, void* stream) {
  if (M <= 0 || N <= 0 || r <= 0) return fail(METIS_ERR_BAD_SHAPE, "empty product %lld x %lld x %lld", (long long)M, (long long)N, (long long)r);
  if (r > 256 || r % 8 != 0 || N % 8 != 0) return fail(METIS_ERR_BAD_SHAPE, "rank %lld must be a multiple of 8 up to 256 and N = %lld a multiple of 8", (long long)r, (long long)N);
  if (int32_t rc = check_bf16_matrix(g, ldg, N, "g")) return rc;
  if (int32_t rc = check_bf16_matrix(ts, ldts, r, "ts")) return rc;
  if (!grad_u || !workspace) return fail(METIS_ERR_BAD_ARGUMENT, "null pointer");
  if (u_dtype != METIS_DTYPE_BF16 && u_dtype != METIS_DTYPE_F32) return fail(METIS_ERR_BAD_ARGUMENT, "unknown u_dtype %d", u_dtype);
  if (ldgu < r) return fail(METIS_ERR_BAD_ARGUMENT, "ldgu %lld < r %lld", (long long)ldgu, (long long)r);
  if (!aligned16(workspace) || workspace_bytes < metis_lowrank_du_workspace_bytes(M, N, r)) return fail(METIS_ERR_WORKSPACE, "workspace too small or misaligned");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const PanelPlan pl = plan_panel(N, r, M);
  float* partial = static_cast<float*>(workspace);
  // dU = G^T ts: both operands hold the contraction (the tokens) in their rows
  if (int32_t rc = launch_panel(g, true, ldg, ts, true, ldts, N, r, M, pl, partial, status, st)) return rc;
  if (u_dtype == METIS_DTYPE_BF16) return launch_sum(partial, pl, N, r, static_cast<__nv_bfloat16*>(grad_u), ldgu, st);
  return launch_sum(partial, pl, N, r, static_cast<float*>(grad_u), ldgu, st);
}

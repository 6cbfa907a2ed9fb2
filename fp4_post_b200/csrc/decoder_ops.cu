// Elementwise pieces of a decoder block around the projections, for inference: rotary embedding of q and k in one launch,
// silu(gate) * up in one.  At decode sizes each torch op of these expressions is a launch of 2-4 us in the block's
// dependent chain (ten for the two rotary embeddings).  Every bf16 rounding of the torch expressions is kept.
#include "common.cuh"

namespace metis {

// out = bf16(bf16(x cos) + bf16(rot(x) sin)), rot(x) = (-x2, x1) of the two halves (rotate-half convention).
// q [tokens, heads_q, D] and k [tokens, heads_k, D], contiguous; cos and sin [positions, D], row t % positions belongs to
// token t.  A thread takes four elements of the first half and their partners in the second: 8-byte accesses.  Bound by
// launch latency at decode sizes (64 tokens of the 7B shape: ten launches, 30 us, before; 3 us) and by memory beyond.
__global__ void __launch_bounds__(256)
rope_pair_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ cos,
                 const __nv_bfloat16* __restrict__ sin, __nv_bfloat16* __restrict__ q_out, __nv_bfloat16* __restrict__ k_out,
                 int64_t tokens, int positions, int heads_q, int heads_k, int D) {
  grid_dependency_wait();
  const int half = D >> 1, per_head = half >> 2, heads = heads_q + heads_k;
  const int64_t total = tokens * heads * per_head;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / per_head;
    const int c = (int)(i - row * per_head) * 4;
    const int64_t t = row / heads;
    const int h = (int)(row - t * heads);
    const bool is_q = h < heads_q;
    const int64_t at = is_q ? (t * heads_q + h) * D : (t * heads_k + (h - heads_q)) * D;
    const __nv_bfloat16* x = (is_q ? q : k) + at;
    __nv_bfloat16* o = (is_q ? q_out : k_out) + at;
    const int64_t pos = (t % positions) * D;
    const uint2 xa = *reinterpret_cast<const uint2*>(x + c), xb = *reinterpret_cast<const uint2*>(x + half + c);
    const uint2 ca = *reinterpret_cast<const uint2*>(cos + pos + c), cb = *reinterpret_cast<const uint2*>(cos + pos + half + c);
    const uint2 sa = *reinterpret_cast<const uint2*>(sin + pos + c), sb = *reinterpret_cast<const uint2*>(sin + pos + half + c);
    const uint32_t x1[2] = {xa.x, xa.y}, x2[2] = {xb.x, xb.y}, c1[2] = {ca.x, ca.y}, c2[2] = {cb.x, cb.y}, s1[2] = {sa.x, sa.y}, s2[2] = {sb.x, sb.y};
    uint32_t o1[2], o2[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      auto as2 = [](const uint32_t& w) { return *reinterpret_cast<const __nv_bfloat162*>(&w); };
      const uint32_t minus_x2 = x2[j] ^ 0x80008000u;
      const __nv_bfloat162 r1 = __hadd2_rn(__hmul2_rn(as2(x1[j]), as2(c1[j])), __hmul2_rn(as2(minus_x2), as2(s1[j])));
      const __nv_bfloat162 r2 = __hadd2_rn(__hmul2_rn(as2(x2[j]), as2(c2[j])), __hmul2_rn(as2(x1[j]), as2(s2[j])));
      o1[j] = *reinterpret_cast<const uint32_t*>(&r1);
      o2[j] = *reinterpret_cast<const uint32_t*>(&r2);
    }
    *reinterpret_cast<uint2*>(o + c) = make_uint2(o1[0], o1[1]);
    *reinterpret_cast<uint2*>(o + half + c) = make_uint2(o2[0], o2[1]);
  }
}

// out = bf16(bf16(silu(gate)) * up), eight elements per thread
__global__ void __launch_bounds__(256)
silu_mul_kernel(const __nv_bfloat16* __restrict__ gate, const __nv_bfloat16* __restrict__ up, __nv_bfloat16* __restrict__ out, int64_t groups) {
  grid_dependency_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < groups; i += (int64_t)gridDim.x * blockDim.x) {
    const uint4 g4 = reinterpret_cast<const uint4*>(gate)[i], u4 = reinterpret_cast<const uint4*>(up)[i];
    const uint32_t g[4] = {g4.x, g4.y, g4.z, g4.w}, u[4] = {u4.x, u4.y, u4.z, u4.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = bf16_lo(g[j]), b = bf16_hi(g[j]);
      const __nv_bfloat162 s = __floats2bfloat162_rn(a / (1.0f + expf(-a)), b / (1.0f + expf(-b)));
      const __nv_bfloat162 r = __hmul2_rn(s, *reinterpret_cast<const __nv_bfloat162*>(&u[j]));
      o[j] = *reinterpret_cast<const uint32_t*>(&r);
    }
    reinterpret_cast<uint4*>(out)[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

}  // namespace metis

using namespace metis;

extern "C" int32_t metis_rope_pair(const void* q, const void* k, const void* cos, const void* sin, void* q_out, void* k_out,
                                   int64_t tokens, int64_t positions, int32_t heads_q, int32_t heads_k, int32_t head_dim, void* stream) {
  if (!q || !k || !cos || !sin || !q_out || !k_out) return fail(METIS_ERR_BAD_ARGUMENT, "null pointer");
  if (tokens <= 0 || positions <= 0 || positions >= ((int64_t)1 << 31) || heads_q <= 0 || heads_k <= 0 || head_dim <= 0 || head_dim % 8 != 0)
    return fail(METIS_ERR_BAD_SHAPE, "tokens, positions and heads must be positive and head_dim a multiple of 8");
  for (const void* p : {q, k, cos, sin, static_cast<const void*>(q_out), static_cast<const void*>(k_out)})
    if (reinterpret_cast<uintptr_t>(p) & 7u) return fail(METIS_ERR_BAD_ALIGNMENT, "tensors must be 8-byte aligned");
  int64_t blocks = ceil_div(tokens * (heads_q + heads_k) * (head_dim / 8), 256);
  const int64_t cap = (int64_t)device_sm_count() * 16;
  if (blocks > cap) blocks = cap;
  METIS_CUDA_OK(launch_overlapped(kLaunchShort, rope_pair_kernel, dim3((unsigned)blocks), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
                                  static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(cos),
                                  static_cast<const __nv_bfloat16*>(sin), static_cast<__nv_bfloat16*>(q_out), static_cast<__nv_bfloat16*>(k_out),
                                  tokens, (int)positions, (int)heads_q, (int)heads_k, (int)head_dim));
  return METIS_OK;
}

extern "C" int32_t metis_silu_mul(const void* gate, const void* up, void* out, int64_t n, void* stream) {
  if (!gate || !up || !out) return fail(METIS_ERR_BAD_ARGUMENT, "null pointer");
  if (n <= 0 || n % 8 != 0) return fail(METIS_ERR_BAD_SHAPE, "the number of elements must be a positive multiple of 8");
  if (!aligned16(gate) || !aligned16(up) || !aligned16(out)) return fail(METIS_ERR_BAD_ALIGNMENT, "tensors must be 16-byte aligned");
  int64_t blocks = ceil_div(n / 8, 256);
  const int64_t cap = (int64_t)device_sm_count() * 16;
  if (blocks > cap) blocks = cap;
  METIS_CUDA_OK(launch_overlapped(kLaunchShort, silu_mul_kernel, dim3((unsigned)blocks), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
                                  static_cast<const __nv_bfloat16*>(gate), static_cast<const __nv_bfloat16*>(up), static_cast<__nv_bfloat16*>(out), n / 8));
  return METIS_OK;
}

// The bf16 ops around the quantised linears of the prefill harness: RMSNorm, and per-head RMSNorm + rotary embedding of
// the query and key heads in place.
//
// Both are bound by HBM: one read and one write of the tensor.  As separate torch ops each was a chain of passes over
// fp32 copies (norm: convert, square, mean, scale, convert back, weight; rotary: four products, two sums, a cat), 20-odd
// launches per layer.
#include "common.cuh"

namespace i4tc {

__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t u) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
}
__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  union { __nv_bfloat16 h[2]; uint32_t u; } p;
  p.h[0] = __float2bfloat16_rn(a); p.h[1] = __float2bfloat16_rn(b);
  return p.u;
}

constexpr int kNormThreads = 256, kNormVecs = 8;   // a row of up to 256 * 8 * 8 = 16384 elements stays in registers

// out = bf16(bf16(x * rsqrt(mean(x^2) + eps)) * w), one block per row.
__global__ void __launch_bounds__(kNormThreads) rmsnorm_kernel(const __nv_bfloat16* __restrict__ x, int K, long long ldx,
                                                               const __nv_bfloat16* __restrict__ w, float eps,
                                                               __nv_bfloat16* __restrict__ out) {
  __shared__ float part[kNormThreads / 32];
  const uint4* src = reinterpret_cast<const uint4*>(x + (long long)blockIdx.x * ldx);
  const int nv = K / 8, t = threadIdx.x;
  uint4 v[kNormVecs];
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < kNormVecs; ++i) {
    const int j = t + i * kNormThreads;
    if (j < nv) {
      v[i] = __ldg(src + j);
      const uint32_t u[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = unpack_bf16x2(u[k]);
        s = fmaf(f.x, f.x, s);
        s = fmaf(f.y, f.y, s);
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((t & 31) == 0) part[t >> 5] = s;
  __syncthreads();
  s = 0.f;
#pragma unroll
  for (int i = 0; i < kNormThreads / 32; ++i) s += part[i];
  const float r = rsqrtf(s / (float)K + eps);
  uint4* dst = reinterpret_cast<uint4*>(out + (long long)blockIdx.x * K);
#pragma unroll
  for (int i = 0; i < kNormVecs; ++i) {
    const int j = t + i * kNormThreads;
    if (j < nv) {
      const uint4 g = __ldg(reinterpret_cast<const uint4*>(w) + j);
      const uint32_t u[4] = {v[i].x, v[i].y, v[i].z, v[i].w}, gw[4] = {g.x, g.y, g.z, g.w};
      uint32_t o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = unpack_bf16x2(u[k]), h = unpack_bf16x2(gw[k]);
        o[k] = pack_bf16x2(bf16_round(f.x * r) * h.x, bf16_round(f.y * r) * h.y);
      }
      dst[j] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// Heads [0, q_heads) with wq and [q_heads, q_heads + k_heads) with wk of every token of qkv (row stride ld, heads of 128):
// normalise, then rotate halves by the token's position (token % seq), in place.  A warp takes a head, a lane four
// consecutive elements; the other half of the rotation is 16 lanes away.  Every bf16 rounding of the separate ops is
// kept, so results differ from theirs by the order of the sum of squares only.
__global__ void __launch_bounds__(256) qk_norm_rope_kernel(__nv_bfloat16* __restrict__ qkv, long long tokens, long long ld, int q_heads,
                                                          int heads, int seq, const __nv_bfloat16* __restrict__ wq,
                                                          const __nv_bfloat16* __restrict__ wk,
                                                          const __nv_bfloat16* __restrict__ cos_t,
                                                          const __nv_bfloat16* __restrict__ sin_t, float eps) {
  const int lane = threadIdx.x & 31;
  const long long item = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (item >= tokens * heads) return;   // whole warps
  const long long tok = item / heads;
  const int head = (int)(item - tok * heads);
  uint2* at = reinterpret_cast<uint2*>(qkv + tok * ld + head * 128) + lane;
  const uint2 u = *at;
  const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y);
  float s = a.x * a.x;
  s = fmaf(a.y, a.y, s); s = fmaf(b.x, b.x, s); s = fmaf(b.y, b.y, s);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const float r = rsqrtf(s * (1.0f / 128.0f) + eps);
  const uint2 gw = __ldg(reinterpret_cast<const uint2*>(head < q_heads ? wq : wk) + lane);
  const float2 g0 = unpack_bf16x2(gw.x), g1 = unpack_bf16x2(gw.y);
  const float x[4] = {bf16_round(bf16_round(a.x * r) * g0.x), bf16_round(bf16_round(a.y * r) * g0.y),
                      bf16_round(bf16_round(b.x * r) * g1.x), bf16_round(bf16_round(b.y * r) * g1.y)};
  const long long row = (tok % seq) * 16 + (lane & 15);   // tables [seq, 64]: 16 uint2 a row
  const uint2 cu = __ldg(reinterpret_cast<const uint2*>(cos_t) + row), su = __ldg(reinterpret_cast<const uint2*>(sin_t) + row);
  const float2 c0 = unpack_bf16x2(cu.x), c1 = unpack_bf16x2(cu.y), s0 = unpack_bf16x2(su.x), s1 = unpack_bf16x2(su.y);
  const float c[4] = {c0.x, c0.y, c1.x, c1.y}, sn[4] = {s0.x, s0.y, s1.x, s1.y};
  const bool low = lane < 16;
  float o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float y = __shfl_xor_sync(0xffffffffu, x[i], 16);
    const float p = bf16_round(x[i] * c[i]), q = bf16_round(y * sn[i]);
    o[i] = low ? p - q : p + q;   // x1 c - x2 s | x2 c + x1 s
  }
  *at = make_uint2(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]));
}

}  // namespace i4tc

using namespace i4tc;

extern "C" int i4tc_rmsnorm(const void* x, int64_t rows, int64_t K, int64_t ldx, const void* weight, float eps, void* out,
                            int device, void* stream) {
  I4TC_REQUIRE(rows >= 0 && K >= 0 && rows < (1ll << 31), I4TC_EINVAL, "bad size");
  if (rows == 0 || K == 0) return I4TC_OK;
  I4TC_REQUIRE(x && weight && out, I4TC_EINVAL, "null pointer");
  I4TC_REQUIRE(K % 8 == 0 && K <= kNormThreads * kNormVecs * 8, I4TC_EUNSUPPORTED, "K must be a multiple of 8 and at most 16384");
  I4TC_REQUIRE(aligned_to(x, 16) && aligned_to(weight, 16) && aligned_to(out, 16) && ldx % 8 == 0, I4TC_EALIGN,
               "rows, weight and output must be 16-byte aligned");
  DeviceGuard guard(device);
  I4TC_CUDA(guard.err);
  rmsnorm_kernel<<<(unsigned)rows, kNormThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), (int)K, ldx, static_cast<const __nv_bfloat16*>(weight), eps,
      static_cast<__nv_bfloat16*>(out));
  I4TC_CUDA(cudaGetLastError());
  return I4TC_OK;
}

extern "C" int i4tc_qk_norm_rope(void* qkv, int64_t tokens, int64_t ld, int64_t q_heads, int64_t k_heads, int64_t seq,
                                 const void* q_weight, const void* k_weight, const void* cos_table, const void* sin_table,
                                 float eps, int device, void* stream) {
  const int64_t heads = q_heads + k_heads;
  I4TC_REQUIRE(tokens >= 0 && q_heads >= 0 && k_heads >= 0 && heads <= 65536 && seq > 0 && seq < (1ll << 31), I4TC_EINVAL, "bad size");
  if (tokens == 0 || heads == 0) return I4TC_OK;
  I4TC_REQUIRE(ld >= heads * 128 && tokens < (1ll << 31) && tokens * heads < (1ll << 33), I4TC_EINVAL, "rows of qkv are shorter than the heads");
  I4TC_REQUIRE(qkv && q_weight && k_weight && cos_table && sin_table, I4TC_EINVAL, "null pointer");
  I4TC_REQUIRE(aligned_to(qkv, 8) && ld % 4 == 0 && aligned_to(q_weight, 8) && aligned_to(k_weight, 8) &&
                   aligned_to(cos_table, 8) && aligned_to(sin_table, 8), I4TC_EALIGN, "operands must be 8-byte aligned");
  DeviceGuard guard(device);
  I4TC_CUDA(guard.err);
  qk_norm_rope_kernel<<<(unsigned)((tokens * heads + 7) / 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<__nv_bfloat16*>(qkv), tokens, ld, (int)q_heads, (int)heads, (int)seq, static_cast<const __nv_bfloat16*>(q_weight),
      static_cast<const __nv_bfloat16*>(k_weight), static_cast<const __nv_bfloat16*>(cos_table),
      static_cast<const __nv_bfloat16*>(sin_table), eps);
  I4TC_CUDA(cudaGetLastError());
  return I4TC_OK;
}

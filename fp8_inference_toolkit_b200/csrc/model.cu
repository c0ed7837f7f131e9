// The bf16 ops around the quantised linears of the prefill harness: RMSNorm, and per-head RMSNorm + rotary embedding of
// the query and key heads in place.
//
// Both are bound by HBM: one read and one write of the tensor.  As separate torch ops each was a chain of passes over
// fp32 copies (norm: convert, square, mean, scale, convert back, weight; rotary: four products, two sums, a cat), 20-odd
// launches per layer.
#include "common.cuh"
#include <type_traits>

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
__global__ void __launch_bounds__(kNormThreads) rmsnorm_kernel(const __nv_bfloat16* x, int K, long long ldx,
                                                               const __nv_bfloat16* w, float eps,
                                                               __nv_bfloat16* __restrict__ out) {
  __shared__ float part[kNormThreads / 32];
  x = pdl_wait(x);
  pdl_fresh(w);
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

// Heads [0, q_heads) with wq and [q_heads, heads) with wk of every token of qkv (row stride ld, heads of 128): normalise, then rotate
// halves by the token's position (token % seq), in place.  A block takes a token (several, where a warp or two hold all heads; few tokens
// are shared by several blocks) and a warp two heads at a time, a lane eight consecutive elements of one; the other half of the rotation
// is 8 lanes away.  Tables and weights stay in registers over the heads.  Every bf16 rounding of the separate ops is kept, so results
// differ from theirs by the order of the sum of squares only (four-element chains, then partners 64, 32, 16, 8 and 4 elements away).
// A warp per head with 8-byte accesses, an index division per head and single conversions was bound by the special-function unit:
// [4096, 40 heads] 38.6 us -> 14.5 (5.8 TB/s of the one read and one write).
constexpr int kRopeWarps = 4;

// Eight bf16 as one 16-byte access, or as two of 8 where an operand is aligned to no more.
template <bool A16>
__device__ __forceinline__ uint4 load_oct(const __nv_bfloat16* p) {
  if constexpr (A16) return *reinterpret_cast<const uint4*>(p);
  const uint2 a = *reinterpret_cast<const uint2*>(p), b = *reinterpret_cast<const uint2*>(p + 4);
  return make_uint4(a.x, a.y, b.x, b.y);
}
template <bool A16>
__device__ __forceinline__ void store_oct(__nv_bfloat16* p, const uint4& v) {
  if constexpr (A16) {
    *reinterpret_cast<uint4*>(p) = v;
  } else {
    *reinterpret_cast<uint2*>(p) = make_uint2(v.x, v.y);
    *reinterpret_cast<uint2*>(p + 4) = make_uint2(v.z, v.w);
  }
}

// WPT: warps of a block that work on the same token.  SPLIT: the block rows of the grid share a token's heads.
template <bool A16, int WPT, bool SPLIT>
__global__ void __launch_bounds__(kRopeWarps * 32) qk_norm_rope_kernel(__nv_bfloat16* qkv, unsigned tokens, long long ld,
                                                                       int q_heads, int heads, int seq,
                                                                       const __nv_bfloat16* wq, const __nv_bfloat16* wk,
                                                                       const __nv_bfloat16* cos_t, const __nv_bfloat16* sin_t,
                                                                       float eps) {
  pdl_wait();
  pdl_fresh(qkv); pdl_fresh(wq); pdl_fresh(wk); pdl_fresh(cos_t); pdl_fresh(sin_t);
  const int lane = threadIdx.x & 31, l = lane & 15;
  const int warps = SPLIT ? (int)gridDim.y * WPT : WPT;   // of the token, and this one among them
  const int warp = (int)(threadIdx.x >> 5) % WPT + (SPLIT ? (int)blockIdx.y * WPT : 0);
  const unsigned tok = blockIdx.x * (kRopeWarps / WPT) + threadIdx.x / (32 * WPT);
  if (WPT < kRopeWarps && tok >= tokens) return;   // whole warps
  __nv_bfloat16* at = qkv + (long long)tok * ld + l * 8;
  const long long row = (long long)(tok % (unsigned)seq) * 64 + (l & 7) * 8;   // tables [seq, 64]
  const uint4 cu = load_oct<A16>(cos_t + row), su = load_oct<A16>(sin_t + row);
  const uint4 gq = load_oct<A16>(wq + l * 8), gk = load_oct<A16>(wk + l * 8);
  const uint32_t c[4] = {cu.x, cu.y, cu.z, cu.w}, sn[4] = {su.x, su.y, su.z, su.w};
  auto b2 = [](uint32_t u) { return *reinterpret_cast<const __nv_bfloat162*>(&u); };
  int h = warp * 2 + (lane >> 4);
  uint4 cur = make_uint4(0u, 0u, 0u, 0u);
  if (h < heads) cur = load_oct<A16>(at + (long long)h * 128);
  for (int h0 = warp * 2; h0 < heads; h0 += warps * 2, h += warps * 2) {   // the same trips for both halves of the warp
    uint4 nxt = make_uint4(0u, 0u, 0u, 0u);
    if (h + warps * 2 < heads) nxt = load_oct<A16>(at + (long long)(h + warps * 2) * 128);
    const uint32_t u[4] = {cur.x, cur.y, cur.z, cur.w};
    float2 f[4];
    float s[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = unpack_bf16x2(u[i]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      s[i] = f[2 * i].x * f[2 * i].x;
      s[i] = fmaf(f[2 * i].y, f[2 * i].y, s[i]);
      s[i] = fmaf(f[2 * i + 1].x, f[2 * i + 1].x, s[i]);
      s[i] = fmaf(f[2 * i + 1].y, f[2 * i + 1].y, s[i]);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
      s[1] += __shfl_xor_sync(0xffffffffu, s[1], o);
    }
    const float r = rsqrtf((s[0] + s[1]) * (1.0f / 128.0f) + eps);
    const bool q = h < q_heads;
    const uint32_t gw[4] = {q ? gq.x : gk.x, q ? gq.y : gk.y, q ? gq.z : gk.z, q ? gq.w : gk.w};
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      // (products of two bf16 are exact in fp32 and a sum of two is never closer to a bf16 tie than fp32 resolves: the packed operations
      // round like fp32 ones rounded to bf16)
      const __nv_bfloat162 x = __hmul2_rn(__floats2bfloat162_rn(f[i].x * r, f[i].y * r), b2(gw[i]));
      const uint32_t mine = *reinterpret_cast<const uint32_t*>(&x);
      const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 8);
      const __nv_bfloat162 p = __hmul2_rn(x, b2(c[i])), t = __hmul2_rn(b2(other), b2(sn[i]));
      const __nv_bfloat162 y = l < 8 ? __hsub2_rn(p, t) : __hadd2_rn(p, t);   // x1 c - x2 s | x2 c + x1 s
      o[i] = *reinterpret_cast<const uint32_t*>(&y);
    }
    if (h < heads) store_oct<A16>(at + (long long)h * 128, make_uint4(o[0], o[1], o[2], o[3]));
    cur = nxt;
  }
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
  I4TC_CUDA(launch_kernel(true, rmsnorm_kernel, dim3((unsigned)rows), kNormThreads, 0, static_cast<cudaStream_t>(stream),
                          static_cast<const __nv_bfloat16*>(x), (int)K, ldx, static_cast<const __nv_bfloat16*>(weight), eps,
                          static_cast<__nv_bfloat16*>(out)));
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
  const bool a16 = aligned_to(qkv, 16) && ld % 8 == 0 && aligned_to(q_weight, 16) && aligned_to(k_weight, 16) &&
                   aligned_to(cos_table, 16) && aligned_to(sin_table, 16);
  // A token's heads: one warp for two, two warps for four, else a block.  [16384, 1 head] 10.0 us with three idle warps a block, 4.6 so.
  // Up to 64 tokens do not fill the device with a block each: one for every eight heads ([1, 72 heads] 3.3 -> 1.5 us).
  const bool split = tokens <= 64 && heads > 8;
  const int wpt = heads <= 2 ? 1 : heads <= 4 ? 2 : kRopeWarps;
  const dim3 grid((unsigned)((tokens * wpt + kRopeWarps - 1) / kRopeWarps), split ? (unsigned)((heads + 7) / 8) : 1u);
  auto pick = [&](auto a) {
    constexpr bool A16 = decltype(a)::value;
    return split      ? qk_norm_rope_kernel<A16, kRopeWarps, true>
           : wpt == 1 ? qk_norm_rope_kernel<A16, 1, false>
           : wpt == 2 ? qk_norm_rope_kernel<A16, 2, false>
                      : qk_norm_rope_kernel<A16, kRopeWarps, false>;
  };
  I4TC_CUDA(launch_kernel(true, a16 ? pick(std::true_type{}) : pick(std::false_type{}), grid, kRopeWarps * 32, 0,
                          static_cast<cudaStream_t>(stream), static_cast<__nv_bfloat16*>(qkv), (unsigned)tokens, ld, (int)q_heads,
                          (int)heads, (int)seq, static_cast<const __nv_bfloat16*>(q_weight), static_cast<const __nv_bfloat16*>(k_weight),
                          static_cast<const __nv_bfloat16*>(cos_table), static_cast<const __nv_bfloat16*>(sin_table), eps));
  return I4TC_OK;
}

// Code arithmetic of the int4 quantisers (shared with the CPU oracle): s = absmax / 7 (IEEE), q = clamp(rint(x / s), -8, 7)
// with IEEE division and round-half-even, q = 0 when absmax == 0.  The returned scale is
// max(s, 1/(7*512)) for activations (int4_quant.cu:97,142) and s or 1.0 (all-zero slice) for
// weights (int4_quant.cu:267).
#pragma once
#include "common.cuh"

namespace i4tc {

__device__ __forceinline__ float min_scale() { return 1.0f / (7.0f * 512.0f); }

// s = RN(absmax / 7)
__device__ __forceinline__ float scale_out(float absmax, float s, int role) {
  if (role == I4TC_ROLE_ACTIVATION) return fmaxf(s, min_scale());
  return absmax == 0.0f ? 1.0f : s;
}

// Eight consecutive elements.  bf16 keeps the raw 128 bits (4 registers) and widens on use; the
// absmax is taken on the packed halves (|x| and max are exact in bf16).  Other types are widened
// at load time.
template <typename T>
struct Vec8 {
  float v[8];
  __device__ __forceinline__ void load(const T* p);
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.f;
  }
  __device__ __forceinline__ float get(int i) const { return v[i]; }
  __device__ __forceinline__ float absmax() const {
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(v[i]));
    return m;
  }
};

template <>
struct Vec8<__nv_bfloat16> {
  uint32_t w[4];
  __device__ __forceinline__ void load(const __nv_bfloat16* p) {
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
    w[0] = u.x; w[1] = u.y; w[2] = u.z; w[3] = u.w;
  }
  __device__ __forceinline__ void zero() { w[0] = w[1] = w[2] = w[3] = 0u; }
  __device__ __forceinline__ float get(int i) const {
    return (i & 1) ? __uint_as_float(w[i >> 1] & 0xFFFF0000u) : __uint_as_float(w[i >> 1] << 16);
  }
  // |x| maxima of the two 16-bit halves, still packed (max and abs are exact in bf16)
  __device__ __forceinline__ __nv_bfloat162 absmax2() const {
    __nv_bfloat162 m = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[0]));
#pragma unroll
    for (int i = 1; i < 4; ++i) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[i])));
    return m;
  }
  __device__ __forceinline__ float absmax() const { return widen_max(absmax2()); }
  // bf16 -> fp32 by moving the 16 bits up (integer pipe; the conversion instruction is much slower)
  static __device__ __forceinline__ float widen_max(__nv_bfloat162 m) {
    const uint32_t b = *reinterpret_cast<const uint32_t*>(&m);
    return fmaxf(__uint_as_float(b << 16), __uint_as_float(b & 0xFFFF0000u));
  }
};

template <>
__device__ __forceinline__ void Vec8<__half>::load(const __half* p) {
  uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
  const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 f = __half22float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
template <>
__device__ __forceinline__ void Vec8<float>::load(const float* p) {
  float4 a = __ldg(reinterpret_cast<const float4*>(p));
  float4 b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

template <typename T>
__device__ __forceinline__ float absmax8(const Vec8<T>& x) { return x.absmax(); }

// Eight codes -> one 32-bit word, element 0 in the lowest nibble.  Exact-division path.
template <typename T>
__device__ __forceinline__ uint32_t pack8_div(const Vec8<T>& x, float s) {
  uint32_t w = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) w |= code4(x.get(i), s) << (4 * i);
  return w;
}

// Reciprocal of the divisor for the fast path.  rcp.approx is within 2^-23 of 1/s; `fast` is false
// when r is not a normal number of moderate size, and then every vector takes the exact path.
struct Recip {
  float r;      // approximately 1 / divisor
  float base;   // absmax (FROM_ABSMAX) or the divisor itself
  bool fast;
};
// FROM_ABSMAX: the divisor is absmax / 7, so r = 7 * rcp(absmax) (within 2^-22 of 1 / RN(absmax/7));
// the IEEE division absmax / 7 is then only needed on the rare exact path.
template <bool FROM_ABSMAX>
__device__ __forceinline__ Recip make_recip(float base) {
  Recip q;
  q.base = base;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q.r) : "f"(base));
  if (FROM_ABSMAX) q.r *= 7.0f;
  q.fast = (q.r > 7.8886090522e-31f) && (q.r < 1.2676506002e30f);  // 2^-100 < r < 2^100
  return q;
}
template <bool FROM_ABSMAX>
__device__ __forceinline__ float exact_divisor(const Recip& q) {
  return FROM_ABSMAX ? __fdiv_rn(q.base, 7.0f) : q.base;
}

// bf16 elements and the divisor RN(absmax / 7): no element has to be decided by itself.
//   With absmax = A * 2^b and x = X * 2^a (A, X 8-bit significands) 7 x / absmax is either exactly k + 0.5 or at least 2.8e-4 away
//   from it (all pairs of significands enumerated).  y = x * r + 40 lies in [32, 64), where fp32 steps by 2^-18: r is within
//   1.8e-7 of 7 / absmax, so an exact half comes out as 40 + h precisely (|error| < 1.2e-6 before rounding) and nothing else
//   does; rounding y to the nearest even integer then gives the code.
//   The definition divides by the ROUNDED quotient s = RN(absmax / 7), so RN(x / s) may miss an exact half by an ulp.  Over all A
//   that happens at |h| = 3.5 only (A = 128, 135, .. 163 and 228, .. 249; each of them has no other halves), where it comes out
//   below 3.5 and the magnitude is 3 and not 4: s_above is that case, and r is then lowered by 2^-17 (5.3e-5 at most, so
//   nothing else changes sides).
// With every half decided by itself behind a branch, half of the warp steps of [16384, 12288] took that branch: 118 us per group
// -> 96 (0.68 -> 0.81 of the copy rate).
struct SnapRecip {
  float r, absmax;
  bool fast;
};
__device__ __forceinline__ SnapRecip make_snap_recip(float absmax, float s) {
  SnapRecip q;
  q.absmax = absmax;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q.r) : "f"(absmax));
  q.r *= 7.0f;
  q.fast = (q.r > 7.8886090522e-31f) && (q.r < 1.2676506002e30f);  // 2^-100 < r < 2^100
  // 3.5 s - absmax / 2 exactly, against half an ulp of 3.5 (2^-23) times s
  const bool s_above = fmaf(3.5f, s, -0.5f * absmax) > s * 1.1920928955078125e-07f;
  if (s_above) q.r *= 1.0f - 7.62939453125e-06f;
  return q;
}
// Slices whose reciprocal is out of range divide (out of line: inlined, this and the other rare paths made the kernels larger
// than the instruction cache, a third of their stalls).
static __device__ __noinline__ uint32_t pack8_div_bf16(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, float s) {
  Vec8<__nv_bfloat16> x;
  x.w[0] = w0; x.w[1] = w1; x.w[2] = w2; x.w[3] = w3;
  return pack8_div(x, s);
}
// Eight codes of a bf16 slice whose absmax gave q; the same words as pack8_div(x, absmax / 7).
__device__ __forceinline__ uint32_t pack8_snap(const Vec8<__nv_bfloat16>& x, const SnapRecip& q, bool zero) {
  if (zero) return 0u;
  if (!q.fast) return pack8_div_bf16(x.w[0], x.w[1], x.w[2], x.w[3], __fdiv_rn(q.absmax, 7.0f));
  constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
  const float2 r2 = make_float2(q.r, q.r), off = make_float2(40.f, 40.f), mg = make_float2(kMagic, kMagic);
  const float2 nmg = make_float2(-kMagic - 32.0f, -kMagic - 32.0f);
  float2 v[4];  // v[i] = (n_i + 8, n_{i+4} + 8)
#pragma unroll
  for (int i = 0; i < 4; ++i)
    v[i] = __fadd2_rn(__fadd2_rn(__ffma2_rn(make_float2(x.get(i), x.get(i + 4)), r2, off), mg), nmg);
  // (lo, hi) = v0 + 16 v1 + 256 v2 + 4096 v3 for elements 0..3 and 4..7: exact, below 2^16
  float2 lh = __ffma2_rn(v[3], make_float2(4096.f, 4096.f),
                         __ffma2_rn(v[2], make_float2(256.f, 256.f), __ffma2_rn(v[1], make_float2(16.f, 16.f), v[0])));
  lh = __fadd2_rn(lh, mg);
  return ((__float_as_uint(lh.x) & 0xFFFFu) | (__float_as_uint(lh.y) << 16)) ^ 0x88888888u;
}

// Exact code (+8) of an element whose quotient lies within ~1e-5 of a rounding boundary h = k + 0.5.
// No division: with a = |x|, e1 = h*s - a is exactly representable (a is that close to h*s), and
// RN(a/s) <= h, = h or >= h is decided by comparing e1 with half an ulp of h times s, also exact.
// rint's tie-to-even then picks k or k+1.  (a/s can never equal the 25-bit midpoint h +- ulp/2.)
__device__ __forceinline__ float exact_tie_code8(float x, float y8, float s) {
  const float a = fabsf(x);
  const float kf = rintf(fabsf(y8 - 8.0f) - 0.5f);      // k >= 0
  const float h = kf + 0.5f;
  const float e1 = fmaf(h, s, -a);                       // exact
  const float pw = __uint_as_float(__float_as_uint(h) & 0x7F800000u);
  const float cs = pw * (s * 5.9604644775390625e-08f);   // (ulp(h) / 2) * s, exact
  const bool odd = (__float2int_rn(kf) & 1) != 0;
  // k even: RN(a/s) <= h rounds to k, above h to k+1.  k odd: RN(a/s) >= h rounds to k+1, below to k.
  const float mag = odd ? ((e1 > cs) ? kf : kf + 1.0f) : ((-e1 > cs) ? kf + 1.0f : kf);
  return copysignf(mag, x) + 8.0f;
}

// Same result as pack8_div, bit for bit, at a fraction of the instructions (packed f32x2 math).
//   y8 = x*r + 8 (one FMA)      u = y8 + 1.5*2^23 rounds y8 to the nearest-even integer n+8 in [0,15]
//   v  = u - 1.5*2^23 = n+8     the eight v's are combined with exact FMAs (16 bits per half)
// |y8 - 8 - RN(x/s)| < 3e-6 for |x/s| <= 8 (r within 2^-22 of 1/s, one rounding in the FMA, one in
// the exact quotient), so unless y8 lies within 1e-5 of a rounding boundary (k + 0.5) the rounded
// integer is that of the exact division.  Elements inside that window (bf16 data produce exact
// ties in about one element per thousand) are decided exactly by exact_tie_code8.
// CLAMP: the caller supplied the divisor, so x/s may leave [-8, 7].
template <typename T, bool CLAMP>
__device__ __forceinline__ uint32_t pack8(const Vec8<T>& x, const Recip& q, bool zero) {
  if (zero) return 0u;
  if (!q.fast) return pack8_div(x, exact_divisor<!CLAMP>(q));
  constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
  constexpr float kThr = 0.5f - 1e-5f;
  const float2 r2 = make_float2(q.r, q.r), eight = make_float2(8.f, 8.f), mg = make_float2(kMagic, kMagic);
  const float2 nmg = make_float2(-kMagic, -kMagic);
  float2 v[4];  // v[i] = (n_i + 8, n_{i+4} + 8)
  float2 e[CLAMP ? 4 : 1];   // CLAMP: e[i] = y8 - v[i] (exact), kept for the rare path
  float worst = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 y8 = __ffma2_rn(make_float2(x.get(i), x.get(i + 4)), r2, eight);
    if (CLAMP) {
      y8.x = fminf(fmaxf(y8.x, 0.0f), 15.0f);
      y8.y = fminf(fmaxf(y8.y, 0.0f), 15.0f);
    }
    v[i] = __fadd2_rn(__fadd2_rn(y8, mg), nmg);
    const float2 d = __ffma2_rn(v[i], make_float2(-1.f, -1.f), y8);
    if (CLAMP) e[i] = d;
    worst = fmaxf(worst, fmaxf(fabsf(d.x), fabsf(d.y)));
  }
  if (!(worst <= kThr)) {
    // rare: some element sits on a rounding boundary
    const float s = exact_divisor<!CLAMP>(q);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (CLAMP) {
        // y8 = v + e exactly (v is y8 rounded to an integer, e the exact remainder): nothing is recomputed
        if (!(fabsf(e[i].x) <= kThr)) v[i].x = exact_tie_code8(x.get(i), v[i].x + e[i].x, s);
        if (!(fabsf(e[i].y) <= kThr)) v[i].y = exact_tie_code8(x.get(i + 4), v[i].y + e[i].y, s);
      } else {
        // (the absmax kernels run at four blocks per SM with 64 registers: recomputing is cheaper than keeping e)
        const float y0 = fmaf(x.get(i), q.r, 8.0f), y1 = fmaf(x.get(i + 4), q.r, 8.0f);
        if (!(fabsf(y0 - v[i].x) <= kThr)) v[i].x = exact_tie_code8(x.get(i), y0, s);
        if (!(fabsf(y1 - v[i].y) <= kThr)) v[i].y = exact_tie_code8(x.get(i + 4), y1, s);
      }
    }
  }
  // (lo, hi) = v0 + 16 v1 + 256 v2 + 4096 v3 for elements 0..3 and 4..7: exact, below 2^16
  float2 lh = __ffma2_rn(v[3], make_float2(4096.f, 4096.f),
                         __ffma2_rn(v[2], make_float2(256.f, 256.f), __ffma2_rn(v[1], make_float2(16.f, 16.f), v[0])));
  lh = __fadd2_rn(lh, mg);
  const uint32_t wl = __float_as_uint(lh.x) & 0xFFFFu;
  const uint32_t wh = __float_as_uint(lh.y) << 16;
  return (wl | wh) ^ 0x88888888u;  // offset-binary nibbles (n+8) -> two's complement
}

// The divisor of an absmax slice and its codes: bf16 slices round by snapping, the other types decide their halves one by one.
template <typename T>
struct AbsmaxCodes {
  Recip q;
  bool zero;
  __device__ __forceinline__ AbsmaxCodes(float absmax, float) : q(make_recip<true>(absmax)), zero(absmax == 0.f) {}
  __device__ __forceinline__ uint32_t word(const Vec8<T>& x) const { return pack8<T, false>(x, q, zero); }
};
template <>
struct AbsmaxCodes<__nv_bfloat16> {
  SnapRecip q;
  bool zero;
  __device__ __forceinline__ AbsmaxCodes(float absmax, float s) : q(make_snap_recip(absmax, s)), zero(absmax == 0.f) {}
  __device__ __forceinline__ uint32_t word(const Vec8<__nv_bfloat16>& x) const { return pack8_snap(x, q, zero); }
};
template <typename T>
struct GivenCodes {
  Recip q;
  __device__ __forceinline__ GivenCodes(float divisor) : q(make_recip<false>(divisor)) {}
  __device__ __forceinline__ uint32_t word(const Vec8<T>& x) const { return pack8<T, true>(x, q, false); }
};

}  // namespace i4tc

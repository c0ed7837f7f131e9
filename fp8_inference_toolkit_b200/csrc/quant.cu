// Fused quantise + pack kernels (bf16/fp16/fp32 -> packed signed int4 + fp32 scales).
//
// One pass over HBM: every element is loaded once with 128-bit loads, stays in registers
// between the absmax reduction (warp shuffles) and the quantise step, and leaves as packed
// 32-bit words (8 codes each).  The reference reads each row twice and uses one 256-thread
// block per 128-element group (int4_native_tc/csrc/int4_quant.cu:100-182, 759-803).
#include "quant_codes.cuh"
#include <type_traits>

namespace i4tc {

// e**t for t clamped to [-87, 87] as a fixed sequence of correctly rounded fp32 operations (never contracted into
// fused multiply-adds): n = rint(t * log2(e)); r = (t - n * ln2_hi) - n * ln2_lo (Cody and Waite's reduction: ln2_hi is ln 2
// cut to 15 significant bits, so n * ln2_hi is exact, ln2_lo the rest); degree-7 Taylor polynomial of r by Horner's rule;
// times 2**n.  A CPU repeats it bit for bit with plain IEEE single-precision arithmetic.
__device__ __forceinline__ float exp_reproducible(float t) {
  t = fminf(fmaxf(t, -87.0f), 87.0f);
  const float n = rintf(__fmul_rn(t, 1.4426950408889634f));
  const float r = __fsub_rn(__fsub_rn(t, __fmul_rn(n, 0.693145751953125f)), __fmul_rn(n, 1.428606765330187045e-06f));
  float p = 1.0f / 5040.0f;
  p = __fadd_rn(__fmul_rn(p, r), 1.0f / 720.0f);
  p = __fadd_rn(__fmul_rn(p, r), 1.0f / 120.0f);
  p = __fadd_rn(__fmul_rn(p, r), 1.0f / 24.0f);
  p = __fadd_rn(__fmul_rn(p, r), 1.0f / 6.0f);
  p = __fadd_rn(__fmul_rn(p, r), 0.5f);
  p = __fadd_rn(__fmul_rn(p, r), 1.0f);
  p = __fadd_rn(__fmul_rn(p, r), 1.0f);
  return __fmul_rn(p, __int_as_float(((int)n + 127) << 23));   // |n| <= 126: an exact power of two
}

// (g * sigmoid(g)) * u with sigmoid(g) = 1 / (1 + exp_reproducible(-g)): the definition of SwiGLU here (out of line, it is rare).
__device__ __noinline__ float silu_mul_reproducible(float g, float u) {
  const float sig = __fdiv_rn(1.0f, __fadd_rn(1.0f, exp_reproducible(-g)));
  return __fmul_rn(__fmul_rn(g, sig), u);
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// bf16(silu(g) * u) of eight elements, bit-identical to bf16(silu_mul_reproducible(g, u)).
// A fast evaluation decides unless its fp32 value lies within 32 ulp of a bf16 rounding boundary (one element in a thousand);
// those elements are evaluated by the definition itself, and so is the whole vector when some |g| > 32 or is not a number.
//   e**-g = 2**(g * hi) * (1 + g * lo), hi = -log2(e) cut to 16 bits (g has 8, so g * hi is exact), lo = ln 2 times the rest:
//   within 2^-22 (the instruction's bound) + 2^-24 (the square of g * lo <= 1.6e-4 is below 2^-26);
//   one reciprocal serves two elements, 1 / a = b * rcp(a b): a, b <= 1 + e**32.
// With the roundings of the steps (3.5 x 2^-23), of the definition's (2 x 2^-23) and its exponential (2 x 2^-23) the two differ
// by less than 11 x 2^-23 relative, 22 ulp.
// Element by element with __expf, an IEEE reciprocal and a branch each: SwiGLU + quantise of [4096, 2 x 12288] 98 us; vectors with the rare paths inlined 79, with them out of line 58.
__device__ __forceinline__ Vec8<__nv_bfloat16> silu_mul8(const Vec8<__nv_bfloat16>& gv, const Vec8<__nv_bfloat16>& uv) {
  constexpr float kHi = -1.4426879882812500f;                 // -log2(e) to 16 bits
  constexpr float kLo = -4.888495152e-06f;                    // (-log2(e) - kHi) * ln 2
  const float2 hi2 = make_float2(kHi, kHi), lo2 = make_float2(kLo, kLo), one = make_float2(1.f, 1.f);
  Vec8<__nv_bfloat16> out;
  float2 y[4];
  uint32_t nearest = 0xFFFFFFFFu;   // two 16-bit minima of (low half - first near value)
  __nv_bfloat162 gmax = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&gv.w[0]));
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 g = make_float2(gv.get(2 * i), gv.get(2 * i + 1)), u = make_float2(uv.get(2 * i), uv.get(2 * i + 1));
    const float2 t = __fmul2_rn(g, hi2);
    const float2 e0 = make_float2(ex2_approx(t.x), ex2_approx(t.y));
    const float2 a = __fadd2_rn(__ffma2_rn(e0, __fmul2_rn(g, lo2), e0), one);
    const float r = rcp_approx(a.x * a.y);
    y[i] = __fmul2_rn(__fmul2_rn(g, make_float2(a.y * r, a.x * r)), u);
    const uint32_t low = __byte_perm(__float_as_uint(y[i].x), __float_as_uint(y[i].y), 0x5410);
    nearest = __viaddmin_u16x2(low, 0x80208020u, nearest);   // low - (0x8000 - 32)
    const __nv_bfloat162 h = __floats2bfloat162_rn(y[i].x, y[i].y);
    out.w[i] = *reinterpret_cast<const uint32_t*>(&h);
    if (i > 0) gmax = __hmax2_nan(gmax, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&gv.w[i])));
  }
  const bool large = !(__low2float(gmax) <= 32.0f && __high2float(gmax) <= 32.0f);
  if ((nearest & 0xFFFFu) <= 64u || (nearest >> 16) <= 64u || large) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool nx = large || (__float_as_uint(y[i].x) & 0xFFFFu) - (0x8000u - 32u) <= 64u;
      const bool ny = large || (__float_as_uint(y[i].y) & 0xFFFFu) - (0x8000u - 32u) <= 64u;
      if (nx) y[i].x = silu_mul_reproducible(gv.get(2 * i), uv.get(2 * i));
      if (ny) y[i].y = silu_mul_reproducible(gv.get(2 * i + 1), uv.get(2 * i + 1));
      const __nv_bfloat162 h = __floats2bfloat162_rn(y[i].x, y[i].y);
      out.w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
  }
  return out;
}

// ------------------------------------------------------------------------------------------
// Grouped kernel.  Block = 8 warps = 8 consecutive rows; each warp owns a 1024-element segment
// of its row (4 x 128-bit loads per lane, all issued before the first use).  A group of
// 8*LPG elements lives in LPG adjacent lanes, so its absmax is log2(LPG) shuffles.
// MODE 0: rows of x.  MODE 1: rows gathered through row_index[r] / index_div.
// MODE 2: input is bf16 [rows, 2*K] laid out [gate | up]; the quantised value is
//         bf16(silu(gate) * up).
// MODE 3: RMSNorm first: the quantised value is bf16(bf16(x * rsqrt(mean(x^2) + eps)) * aux[k]); a warp then
//         needs its whole row (the grid is not split along K).
// GIVEN: divisors come from `given_scale` (group-major) instead of the absmax.
// ------------------------------------------------------------------------------------------
constexpr int kQRows = 8;
constexpr int kQVecs = 4;                 // 8-element vectors per lane per segment
constexpr int kQLane = 8 * kQVecs;        // 32 consecutive elements per lane
constexpr int kQSeg = 32 * kQLane;        // 1024 elements per warp per segment

template <typename T, int MODE>
__device__ __forceinline__ void load_segment(Vec8<T> (&v)[kQVecs], const T* src, int k, int K, bool row_ok,
                                             const T* aux = nullptr, float row_factor = 0.f) {
  // k = first element of this lane; K % 32 == 0, so the lane's 32 elements are all in range or none
  if (row_ok && k < K) {
#pragma unroll
    for (int j = 0; j < kQVecs; ++j) {
      if constexpr (MODE == 2) {
        Vec8<T> g, u;
        g.load(src + k + 8 * j);
        u.load(src + K + k + 8 * j);
        v[j] = silu_mul8(g, u);
      } else if constexpr (MODE == 3) {
        // RMSNorm in front of the quantiser: bf16(bf16(x * inv_rms) * weight), the roundings of an unfused
        // normalisation that works in fp32 and returns the input's type
        Vec8<T> xv, wv;
        xv.load(src + k + 8 * j);
        wv.load(aux + k + 8 * j);
        // two elements per conversion (one at a time they run on the special-function unit, 40 % busy then); a product of two bf16
        // is exact in fp32, so the packed multiply rounds like the separate one
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __nv_bfloat162 n = __floats2bfloat162_rn(xv.get(2 * i) * row_factor, xv.get(2 * i + 1) * row_factor);
          const __nv_bfloat162 h = __hmul2_rn(n, *reinterpret_cast<const __nv_bfloat162*>(&wv.w[i]));
          v[j].w[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
      } else {
        v[j].load(src + k + 8 * j);
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < kQVecs; ++j) v[j].zero();
  }
}

template <typename T>
__device__ __forceinline__ float absmax_of(const Vec8<T> (&v)[kQVecs]) {
  float m = 0.f;
#pragma unroll
  for (int j = 0; j < kQVecs; ++j) m = fmaxf(m, v[j].absmax());
  return m;
}
template <>
__device__ __forceinline__ float absmax_of<__nv_bfloat16>(const Vec8<__nv_bfloat16> (&v)[kQVecs]) {
  __nv_bfloat162 m = v[0].absmax2();
#pragma unroll
  for (int j = 1; j < kQVecs; ++j) m = __hmax2(m, v[j].absmax2());
  return Vec8<__nv_bfloat16>::widen_max(m);
}

// Block = 8 warps = 8 consecutive rows (the warps are independent).  In a segment every lane owns 32 consecutive elements
// (64 bytes of bf16), so a group of GS elements is LPG = GS/32 adjacent lanes: its absmax costs
// log2(LPG) shuffles, its reciprocal is formed once per lane, and each lane leaves 16 packed bytes
// with one 128-bit store.  The block walks `segs_per_block` segments of its rows and loads segment
// s+1 while it quantises segment s.
// OUTMAP (expert-parallel MoE): output row r goes to row out.row_map[r] (skipped when negative) of a layout given by
// byte / float strides instead of the group-major default, and rows at or beyond *out.rows_dev are skipped.
struct QuantOutMap {
  const int32_t* row_map;   // nullptr: identity
  const int32_t* rows_dev;  // nullptr: all `rows`
  long long pk_gstride, pk_rstride;   // bytes between groups / rows of the packed output
  long long sc_gstride, sc_rstride;   // floats between groups / rows of the scale output
  // Peer destinations (nullptr: one local buffer).  Mapped row m lies in block m / block_rows; that block's rows go
  // to the buffer at dest_bases[block] (another GPU's memory, written with plain stores over NVLink), where this
  // rank's block is number my_block: row my_block * block_rows + m % block_rows.  scale_offset = bytes from a row's
  // codes to its scales.
  const unsigned long long* dest_bases;
  int block_rows, my_block;
  long long scale_offset;
};

// Rows (= warps) of a block.  MODE 3 keeps a warp on one row for two passes, so its grid is short: [4096, 4096] is 512 blocks of
// eight warps, 1.15 waves of what fits; half the block and 64 registers (32 warps an SM) make it one wave: with packed conversions
// 21.4 -> 16.3 us.
template <int MODE>
__host__ __device__ constexpr int quant_rows() { return MODE == 3 ? 4 : kQRows; }

template <typename T, int LPG, int MODE, bool GIVEN, bool OUTMAP = false>
__global__ void __launch_bounds__(quant_rows<MODE>() * 32, MODE == 3 ? 8 : MODE == 2 ? 3 : 1) quant_grouped_kernel(
    const T* __restrict__ x, int64_t rows, int K, int64_t ldx, const int32_t* row_index,
    int index_div, int64_t src_rows, const float* given_scale, uint8_t* __restrict__ packed,
    float* __restrict__ scale, int role, int segs_per_block, const T* aux, float eps,
    QuantOutMap out = QuantOutMap{nullptr, nullptr, 0, 0, 0, 0, nullptr, 1, 0, 0}) {
  constexpr int GS = LPG * kQLane;
  if (MODE == 0) pdl_trigger();   // (the GEMM behind it may start)
  if (MODE >= 2) {   // launched so that it starts under the end of the kernel in front of it
    x = pdl_wait(x);
    pdl_fresh(aux); pdl_fresh(row_index); pdl_fresh(given_scale);
    pdl_trigger();
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t r = (int64_t)blockIdx.x * quant_rows<MODE>() + warp;
  bool row_ok = r < rows;
  int64_t orow = r;
  if (OUTMAP) {
    if (out.rows_dev != nullptr && r >= (int64_t)__ldg(out.rows_dev)) row_ok = false;
    if (row_ok && out.row_map != nullptr) {
      orow = __ldg(out.row_map + r);
      if (orow < 0) row_ok = false;
    }
  }
  const int nseg = (K + kQSeg - 1) / kQSeg;
  const int seg_begin = blockIdx.y * segs_per_block;
  const int seg_end = min(nseg, seg_begin + segs_per_block);

  const T* src = nullptr;
  bool src_ok = row_ok;   // MODE 1: false for a pair index that names no row of x (such a row is quantised as zeros)
  if (row_ok) {
    int64_t sr = r;
    if (MODE == 1) {
      const int idx = row_index[r];
      sr = idx / index_div;
      src_ok = idx >= 0 && sr < src_rows;
    }
    if (src_ok) src = x + sr * ldx;
  }
  float row_factor = 0.f;
  if (MODE == 3) {
    // first pass over the row: sum of squares in fp32, the next segment loaded under this one's chain (the second pass below
    // hits L1/L2)
    float ss = 0.f;
    Vec8<T> c0[kQVecs], c1[kQVecs];
    load_segment<T, 0>(c0, src, lane * kQLane, K, row_ok);
    for (int k = lane * kQLane; k - lane * kQLane < K; k += kQSeg) {
      load_segment<T, 0>(c1, src, k + kQSeg, K, row_ok);
#pragma unroll
      for (int j = 0; j < kQVecs; ++j) {
#pragma unroll
        for (int i = 0; i < 8; ++i) ss = fmaf(c0[j].get(i), c0[j].get(i), ss);   // (zeros past the row's end add nothing)
      }
#pragma unroll
      for (int j = 0; j < kQVecs; ++j) c0[j] = c1[j];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    // correctly rounded division, addition and reciprocal square root: a CPU can repeat the row statistic exactly
    row_factor = __frsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)K), eps));
  }
  Vec8<T> cur[kQVecs], nxt[kQVecs];
  load_segment<T, MODE>(cur, src, seg_begin * kQSeg + lane * kQLane, K, src_ok, aux, row_factor);
  for (int seg = seg_begin; seg < seg_end; ++seg) {
    const int k = seg * kQSeg + lane * kQLane;
    if (seg + 1 < seg_end) load_segment<T, MODE>(nxt, src, k + kQSeg, K, src_ok, aux, row_factor);
    const bool ok = row_ok && k < K;
    const int g = k / GS;
    uint4 w;
    if constexpr (GIVEN) {
      const GivenCodes<T> codes(ok ? __ldg(given_scale + (int64_t)g * rows + r) : 1.f);
      w = make_uint4(codes.word(cur[0]), codes.word(cur[1]), codes.word(cur[2]), codes.word(cur[3]));
    } else {
      float absmax = absmax_of(cur);
#pragma unroll
      for (int o = 1; o < LPG; o <<= 1) absmax = fmaxf(absmax, __shfl_xor_sync(0xffffffffu, absmax, o));
      const float s = __fdiv_rn(absmax, 7.0f);
      const AbsmaxCodes<T> codes(absmax, s);
      // one lane per group writes the scale; neighbouring rows fill the same 32-byte sector from other warps
      if (ok && (lane % LPG) == 0) {
        if (OUTMAP) {
          float* sdst = scale + (int64_t)g * out.sc_gstride + orow * out.sc_rstride;
          if (out.dest_bases != nullptr) {
            const int blk = (int)(orow / out.block_rows);
            const int64_t prow = (int64_t)out.my_block * out.block_rows + (orow - (int64_t)blk * out.block_rows);
            sdst = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(out.dest_bases[blk]) + prow * out.pk_rstride +
                                            out.scale_offset) + (int64_t)g * out.sc_gstride;
          }
          *sdst = scale_out(absmax, s, role);
        } else {
          scale[(int64_t)g * rows + r] = scale_out(absmax, s, role);
        }
      }
      w = make_uint4(codes.word(cur[0]), codes.word(cur[1]), codes.word(cur[2]), codes.word(cur[3]));
    }
    if (ok) {
      uint8_t* dst = OUTMAP ? packed + (int64_t)g * out.pk_gstride + orow * out.pk_rstride + (lane % LPG) * 16
                            : packed + ((int64_t)g * rows + r) * (GS / 2) + (lane % LPG) * 16;
      if (OUTMAP && out.dest_bases != nullptr) {
        const int blk = (int)(orow / out.block_rows);
        const int64_t prow = (int64_t)out.my_block * out.block_rows + (orow - (int64_t)blk * out.block_rows);
        dst = reinterpret_cast<uint8_t*>(out.dest_bases[blk]) + prow * out.pk_rstride + (int64_t)g * out.pk_gstride +
              (lane % LPG) * 16;
      }
      *reinterpret_cast<uint4*>(dst) = w;
    }
#pragma unroll
    for (int j = 0; j < kQVecs; ++j) cur[j] = nxt[j];
  }
}

// Tokens quantised once and written to every row that wants them: token t's codes and scales go to rows inv[t * top_k + j] of the
// group-major [G, R, 64] / [G, R] destination (none for an index that is negative or past it).  The layout of the kernel above, group size 128.
// As a quantiser and a copy of its packed rows [4096 tokens, 2048] x 8 took 6.4 + 13.8 us and two launches; here 11.4.
__global__ void __launch_bounds__(256) quant_fanout_kernel(const __nv_bfloat16* x, int64_t rows, int K, int64_t ldx,
                                                           const int32_t* inv, int top_k, int64_t R,
                                                           uint8_t* __restrict__ packed, float* __restrict__ scale) {
  pdl_wait();
  pdl_fresh(x);
  pdl_fresh(inv);
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t r = (int64_t)blockIdx.x * kQRows + warp;
  if (r >= rows) return;   // the whole warp
  const int k = blockIdx.y * kQSeg + lane * kQLane;
  Vec8<__nv_bfloat16> v[kQVecs];
  load_segment<__nv_bfloat16, 0>(v, x + r * ldx, k, K, true);
  float absmax = absmax_of(v);
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) absmax = fmaxf(absmax, __shfl_xor_sync(0xffffffffu, absmax, o));
  const float s = __fdiv_rn(absmax, 7.0f);
  const AbsmaxCodes<__nv_bfloat16> codes(absmax, s);
  const uint4 w = make_uint4(codes.word(v[0]), codes.word(v[1]), codes.word(v[2]), codes.word(v[3]));
  const float sc = scale_out(absmax, s, I4TC_ROLE_ACTIVATION);
  const int64_t g = k / 128;
  for (int j0 = 0; j0 < top_k; j0 += 32) {
    const int mine = j0 + lane < top_k ? __ldg(inv + r * top_k + j0 + lane) : -1;
    for (int j = 0; j < min(32, top_k - j0); ++j) {
      const int64_t pos = __shfl_sync(0xffffffffu, mine, j);
      if ((uint64_t)pos >= (uint64_t)R || k >= K) continue;
      *reinterpret_cast<uint4*>(packed + (g * R + pos) * 64 + (lane & 3) * 16) = w;
      if ((lane & 3) == 0) scale[g * R + pos] = sc;
    }
  }
}

// ------------------------------------------------------------------------------------------
// Clipped symmetric and asymmetric per-group quantisers on the layout of the grouped kernel above (a lane owns 32
// consecutive elements, a group is LPG adjacent lanes, 128-bit loads and stores, next segment loaded while this one is
// quantised).  Arithmetic per group, IEEE fp32:
//   t = max|x| * clip
//   symmetric:  s = t / 7;  code = clamp(rint(x / s), -8, 7), 0 when s == 0;  scale = max(s, 1/(7*512))
//   asymmetric: c = clamp(x, -t, t);  s = max((max c - min c) / 15, 1/(7*512));  azp = clamp(rint(-min c / s), 0, 15);
//               u = clamp(rint(c / s + azp), 0, 15);  stored nibble = u - 8;  azp_adj = 8 - azp
// ------------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void minmax_of(const Vec8<T> (&v)[kQVecs], float& mn, float& mx) {
  mn = INFINITY;
  mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < kQVecs; ++j) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      mn = fminf(mn, v[j].v[i]);
      mx = fmaxf(mx, v[j].v[i]);
    }
  }
}
template <>
__device__ __forceinline__ void minmax_of<__nv_bfloat16>(const Vec8<__nv_bfloat16> (&v)[kQVecs], float& mn, float& mx) {
  // min and max of packed bf16 halves are exact
  __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&v[0].w[0]), hi = lo;
#pragma unroll
  for (int j = 0; j < kQVecs; ++j) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&v[j].w[i]);
      lo = __hmin2(lo, h);
      hi = __hmax2(hi, h);
    }
  }
  const uint32_t bl = *reinterpret_cast<const uint32_t*>(&lo), bh = *reinterpret_cast<const uint32_t*>(&hi);
  mn = fminf(__uint_as_float(bl << 16), __uint_as_float(bl & 0xFFFF0000u));
  mx = fmaxf(__uint_as_float(bh << 16), __uint_as_float(bh & 0xFFFF0000u));
}

// Parameters of one asymmetric group, the same in all its lanes.
struct AsymGroup {
  float thr, s, r, azp;   // clip range, step, ~1/step, zero point
  float ylo, yhi;         // images of -thr / +thr under y = c * r + azp, intersected with [0, 15]
  bool fast;
};

// Eight unsigned codes u (stored as u - 8).  Fast path: y = x * r + azp in one FMA.  The FMA is monotone in x, so
// clamping y to [y(-thr), y(thr)] equals clamping x first; intersected with [0, 15] that is one clamp per element.
// For |c / s| < 64 the FMA lies within 2e-5 of RN(RN(c / s) + azp), so outside 1e-4 of a rounding boundary both round to
// the same integer; for |c / s| >= 64 both saturate on the same side.  Elements inside the window take the IEEE
// division.
template <typename T>
__device__ __forceinline__ uint32_t pack8_asym(const Vec8<T>& x, const AsymGroup& q) {
  constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
  constexpr float kThr = 0.5f - 1e-4f;
  const float2 r2 = make_float2(q.r, q.r), az = make_float2(q.azp, q.azp), mg = make_float2(kMagic, kMagic);
  const float2 nmg = make_float2(-kMagic, -kMagic);
  float2 v[4], y[4];
  float worst = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    y[i] = __ffma2_rn(make_float2(x.get(i), x.get(i + 4)), r2, az);
    y[i].x = fminf(fmaxf(y[i].x, q.ylo), q.yhi);
    y[i].y = fminf(fmaxf(y[i].y, q.ylo), q.yhi);
    v[i] = __fadd2_rn(__fadd2_rn(y[i], mg), nmg);
    const float2 e = __ffma2_rn(v[i], make_float2(-1.f, -1.f), y[i]);
    worst = fmaxf(worst, fmaxf(fabsf(e.x), fabsf(e.y)));
  }
  if (!q.fast || !(worst <= kThr)) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (!q.fast || !(fabsf(y[i].x - v[i].x) <= kThr)) {
        const float c = fminf(fmaxf(x.get(i), -q.thr), q.thr);
        v[i].x = fminf(fmaxf(rintf(__fadd_rn(__fdiv_rn(c, q.s), q.azp)), 0.0f), 15.0f);
      }
      if (!q.fast || !(fabsf(y[i].y - v[i].y) <= kThr)) {
        const float c = fminf(fmaxf(x.get(i + 4), -q.thr), q.thr);
        v[i].y = fminf(fmaxf(rintf(__fadd_rn(__fdiv_rn(c, q.s), q.azp)), 0.0f), 15.0f);
      }
    }
  }
  float2 lh = __ffma2_rn(v[3], make_float2(4096.f, 4096.f),
                         __ffma2_rn(v[2], make_float2(256.f, 256.f), __ffma2_rn(v[1], make_float2(16.f, 16.f), v[0])));
  lh = __fadd2_rn(lh, mg);
  const uint32_t wl = __float_as_uint(lh.x) & 0xFFFFu;
  const uint32_t wh = __float_as_uint(lh.y) << 16;
  return (wl | wh) ^ 0x88888888u;   // u - 8 as a two's-complement nibble is u ^ 8
}

// x / f of one element (out of line: only elements out of the range below come here).
__device__ __noinline__ float div_exact(float x, float f) { return __fdiv_rn(x, f); }

// v[i] = RN(x[i] / f[i]) for eight 16-bit elements and factors.  An approximate quotient q0 = x * y (y ~ 1 / f within 2^-23) and its
// remainder r = x - q0 * f, exact in one fused multiply-add, give q = RN(q0 + r * y) (Markstein's correction), which is
// off x / f by less than 2^-45 relative before the rounding; a quotient of significands of at most 11 bits is no closer than
// 2^-36 to the middle between two fp32 numbers, so q is the correctly rounded one.  Elements and factors whose quotient or remainder
// could leave the normal range, zeros of the factor, infinities and NaN divide.
// [1500, 4096] asymmetric: a division per element in quant_ext_kernel 17.1 us, in this kernel 17.2, corrected reciprocals 11.5.
template <typename T>
__device__ __forceinline__ void smooth_div8(const uint4& xu, const uint4& fu, float (&v)[8]) {
  constexpr bool BF = std::is_same<T, __nv_bfloat16>::value;
  // magnitudes as integers: bf16 |x| in {0} or [2^-40, 2^60], |f| in [2^-40, 2^40]; fp16 anything finite, |f| > 0
  constexpr uint32_t kXLo = BF ? 0x2B80u : 1u, kXHi = BF ? 0x5D80u : 0x7BFFu, kFLo = BF ? 0x2B80u : 1u, kFHi = BF ? 0x5380u : 0x7BFFu;
  const uint32_t xw[4] = {xu.x, xu.y, xu.z, xu.w}, fw[4] = {fu.x, fu.y, fu.z, fu.w};
  uint32_t xlo = 0xFFFFFFFFu, xhi = 0u, flo = 0xFFFFFFFFu, fhi = 0u;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t xa = xw[i] & 0x7FFF7FFFu, fa = fw[i] & 0x7FFF7FFFu;
    xlo = __viaddmin_u16x2(xa, 0xFFFFFFFFu, xlo);   // (a zero becomes the largest value)
    xhi = __vmaxu2(xa, xhi);
    flo = __vminu2(fa, flo);
    fhi = __vmaxu2(fa, fhi);
    float2 x, f;
    if constexpr (BF) {
      x = make_float2(__uint_as_float(xw[i] << 16), __uint_as_float(xw[i] & 0xFFFF0000u));
      f = make_float2(__uint_as_float(fw[i] << 16), __uint_as_float(fw[i] & 0xFFFF0000u));
    } else {
      x = __half22float2(*reinterpret_cast<const __half2*>(&xw[i]));
      f = __half22float2(*reinterpret_cast<const __half2*>(&fw[i]));
    }
    const float2 y = make_float2(rcp_approx(f.x), rcp_approx(f.y));
    const float2 q0 = __fmul2_rn(x, y);
    const float2 r = __ffma2_rn(make_float2(-q0.x, -q0.y), f, x);
    const float2 q = __ffma2_rn(r, y, q0);
    v[2 * i] = q.x;
    v[2 * i + 1] = q.y;
  }
  const bool ok = (xlo & 0xFFFFu) + 1u >= kXLo && (xlo >> 16) + 1u >= kXLo &&
                  (xhi & 0xFFFFu) <= kXHi && (xhi >> 16) <= kXHi && (flo & 0xFFFFu) >= kFLo && (flo >> 16) >= kFLo &&
                  (fhi & 0xFFFFu) <= kFHi && (fhi >> 16) <= kFHi;
  if (!ok) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float x, f;
      const uint32_t xi = (xw[i / 2] >> (16 * (i & 1))) & 0xFFFFu, fi = (fw[i / 2] >> (16 * (i & 1))) & 0xFFFFu;
      if constexpr (BF) {
        x = __uint_as_float(xi << 16);
        f = __uint_as_float(fi << 16);
      } else {
        x = __half2float(__ushort_as_half((unsigned short)xi));
        f = __half2float(__ushort_as_half((unsigned short)fi));
      }
      v[i] = div_exact(x, f);
    }
  }
}

template <typename T>
constexpr uint32_t kOnes = std::is_same<T, __nv_bfloat16>::value ? 0x3F803F80u : 0x3C003C00u;   // 1.0 twice

// SMOOTH: every element is divided (IEEE, fp32) by its channel's factor first, and fp32 values are quantised.
template <typename T, int LPG, bool ASYM, bool SMOOTH>
__global__ void __launch_bounds__(256) quant_grouped_ext_kernel(const T* __restrict__ x, int64_t rows, int K,
                                                                int64_t ldx, float clip, const T* __restrict__ smooth,
                                                                uint8_t* __restrict__ packed, float* __restrict__ scale,
                                                                float* __restrict__ azp_adj, int segs_per_block) {
  pdl_trigger();
  using V = typename std::conditional<SMOOTH, float, T>::type;
  constexpr int GS = LPG * kQLane;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t r = (int64_t)blockIdx.x * kQRows + warp;
  const bool row_ok = r < rows;
  const int nseg = (K + kQSeg - 1) / kQSeg;
  const int seg_begin = blockIdx.y * segs_per_block;
  const int seg_end = min(nseg, seg_begin + segs_per_block);
  const T* src = row_ok ? x + r * ldx : nullptr;
  using S = typename std::conditional<SMOOTH, __nv_bfloat16, T>::type;   // SMOOTH keeps 16-bit words, whatever they hold
  Vec8<S> cur[kQVecs], nxt[kQVecs];
  const S* ssrc = reinterpret_cast<const S*>(src);
  load_segment<S, 0>(cur, ssrc, seg_begin * kQSeg + lane * kQLane, K, row_ok);
  for (int seg = seg_begin; seg < seg_end; ++seg) {
    const int k = seg * kQSeg + lane * kQLane;
    if (seg + 1 < seg_end) load_segment<S, 0>(nxt, ssrc, k + kQSeg, K, row_ok);
    const bool ok = row_ok && k < K;
    const int g = k / GS;
    float mn, mx;
    Vec8<V> val[kQVecs];
    if constexpr (SMOOTH) {
#pragma unroll
      for (int j = 0; j < kQVecs; ++j) {
        uint4 f = make_uint4(kOnes<T>, kOnes<T>, kOnes<T>, kOnes<T>);   // (past the row's end: zeros over ones)
        if (k < K) f = __ldg(reinterpret_cast<const uint4*>(smooth + k + 8 * j));
        smooth_div8<T>(make_uint4(cur[j].w[0], cur[j].w[1], cur[j].w[2], cur[j].w[3]), f, val[j].v);
      }
    } else {
#pragma unroll
      for (int j = 0; j < kQVecs; ++j) val[j] = cur[j];
    }
    minmax_of(val, mn, mx);
#pragma unroll
    for (int o = 1; o < LPG; o <<= 1) {
      mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    const float thr = __fmul_rn(fmaxf(-mn, mx), clip);
    uint4 w;
    if (ASYM) {
      AsymGroup q;
      q.thr = thr;
      const float cmn = fminf(fmaxf(mn, -thr), thr), cmx = fminf(fmaxf(mx, -thr), thr);
      q.s = fmaxf(__fdiv_rn(__fsub_rn(cmx, cmn), 15.0f), min_scale());
      q.azp = fminf(fmaxf(rintf(__fdiv_rn(-cmn, q.s)), 0.0f), 15.0f);
      asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q.r) : "f"(q.s));
      q.fast = (q.r > 7.8886090522e-31f) && (q.r < 1.2676506002e30f);
      q.ylo = fmaxf(fmaf(-thr, q.r, q.azp), 0.0f);
      q.yhi = fminf(fmaf(thr, q.r, q.azp), 15.0f);
      if (ok && (lane % LPG) == 0) {
        scale[(int64_t)g * rows + r] = q.s;
        azp_adj[(int64_t)g * rows + r] = 8.0f - q.azp;
      }
      w.x = pack8_asym<V>(val[0], q);
      w.y = pack8_asym<V>(val[1], q);
      w.z = pack8_asym<V>(val[2], q);
      w.w = pack8_asym<V>(val[3], q);
    } else {
      const float s = __fdiv_rn(thr, 7.0f);
      const bool zero = !(s > 0.0f);
      const Recip q = make_recip<false>(zero ? 1.0f : s);
      if (ok && (lane % LPG) == 0) scale[(int64_t)g * rows + r] = fmaxf(s, min_scale());
      w.x = pack8<V, true>(val[0], q, zero);
      w.y = pack8<V, true>(val[1], q, zero);
      w.z = pack8<V, true>(val[2], q, zero);
      w.w = pack8<V, true>(val[3], q, zero);
    }
    if (ok) *reinterpret_cast<uint4*>(packed + ((int64_t)g * rows + r) * (GS / 2) + (lane % LPG) * 16) = w;
#pragma unroll
    for (int j = 0; j < kQVecs; ++j) cur[j] = nxt[j];
  }
}

template <typename T, bool ASYM, bool SMOOTH = false>
static int launch_grouped_ext_t(const T* x, int64_t rows, int64_t K, int64_t ldx, int gs, float clip, const T* smooth, uint8_t* packed,
                                float* scale, float* azp_adj, cudaStream_t st) {
  const int64_t row_blocks = (rows + kQRows - 1) / kQRows;
  const int nseg = (int)((K + kQSeg - 1) / kQSeg);
  int spb = nseg;
  if (row_blocks < 2048) spb = (int)((int64_t)nseg * row_blocks / 2048);
  if (spb < 1) spb = 1;
  dim3 grid((unsigned)row_blocks, (unsigned)((nseg + spb - 1) / spb));
  I4TC_REQUIRE(grid.y <= 65535, I4TC_EINVAL, "K=%lld too large for the grouped quantiser", (long long)K);
#define I4TC_LAUNCH_E(LPG) \
  quant_grouped_ext_kernel<T, LPG, ASYM, SMOOTH><<<grid, 256, 0, st>>>(x, rows, (int)K, ldx, clip, smooth, packed, scale, azp_adj, spb)
  switch (gs) {
    case 64: I4TC_LAUNCH_E(2); break;
    case 128: I4TC_LAUNCH_E(4); break;
    case 256: I4TC_LAUNCH_E(8); break;
    default: return fail(I4TC_EUNSUPPORTED, "group_size=%d not supported (64, 128 or 256)", gs);
  }
#undef I4TC_LAUNCH_E
  I4TC_CUDA(cudaGetLastError());
  return I4TC_OK;
}

// Whether the vectorised kernel can take this call: 16-byte aligned rows, smoothing factors and outputs (it moves 128 bits per lane).
bool grouped_ext_fast_ok(const void* x, int64_t ldx, const void* smooth, const uint8_t* packed) {
  return aligned_to(x, 16) && (ldx * 2) % 16 == 0 && aligned_to(smooth, 16) && aligned_to(packed, 16);
}

template <typename T>
static int launch_grouped_ext_d(bool asym, const void* x, int64_t rows, int64_t K, int64_t ldx, int gs, float clip, const void* smooth,
                                uint8_t* packed, float* scale, float* azp_adj, cudaStream_t st) {
  const T* p = static_cast<const T*>(x);
  const T* f = static_cast<const T*>(smooth);
  if (!asym) return launch_grouped_ext_t<T, false>(p, rows, K, ldx, gs, clip, nullptr, packed, scale, azp_adj, st);
  return f == nullptr ? launch_grouped_ext_t<T, true>(p, rows, K, ldx, gs, clip, nullptr, packed, scale, azp_adj, st)
                      : launch_grouped_ext_t<T, true, true>(p, rows, K, ldx, gs, clip, f, packed, scale, azp_adj, st);
}

int launch_grouped_ext(bool asym, const void* x, int dtype, int64_t rows, int64_t K, int64_t ldx, int gs, float clip,
                       const void* smooth, uint8_t* packed, float* scale, float* azp_adj, cudaStream_t st) {
  if (dtype == I4TC_BF16) return launch_grouped_ext_d<__nv_bfloat16>(asym, x, rows, K, ldx, gs, clip, smooth, packed, scale, azp_adj, st);
  if (dtype == I4TC_FP16) return launch_grouped_ext_d<__half>(asym, x, rows, K, ldx, gs, clip, smooth, packed, scale, azp_adj, st);
  return fail(I4TC_EUNSUPPORTED, "input must be bf16 or fp16 (dtype %d)", dtype);
}

// ------------------------------------------------------------------------------------------
// Row-wise kernel.  One 256-thread block per row; the row is cached in registers
// (NCH chunks of 2048 elements, 8 per thread per chunk), so HBM is read once.
// ------------------------------------------------------------------------------------------
// TRIGGER: a GEMM behind it may start early.
template <typename T, int NCH, bool GIVEN, bool TRIGGER>
__global__ void __launch_bounds__(256) quant_rowwise_kernel(const T* __restrict__ x, int K, int64_t ldx,
                                                            const float* __restrict__ given_scale,
                                                            uint8_t* __restrict__ packed,
                                                            float* __restrict__ scale, int role) {
  __shared__ float s_max[8];
  if (TRIGGER) pdl_trigger();
  const int64_t r = blockIdx.x;
  const T* src = x + r * ldx;
  const int t = threadIdx.x;
  Vec8<T> v[NCH];
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int k = c * 2048 + t * 8;
    if (k < K) v[c].load(src + k); else v[c].zero();
  }
  uint8_t* dst = packed + r * (int64_t)(K / 2);
  auto store = [&](const auto& codes) {
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int k = c * 2048 + t * 8;
      if (k < K) *reinterpret_cast<uint32_t*>(dst + k / 2) = codes.word(v[c]);
    }
  };
  if constexpr (GIVEN) {
    store(GivenCodes<T>(__ldg(given_scale + r)));
  } else {
    float absmax = 0.f;
#pragma unroll
    for (int c = 0; c < NCH; ++c) absmax = fmaxf(absmax, absmax8(v[c]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) absmax = fmaxf(absmax, __shfl_xor_sync(0xffffffffu, absmax, o));
    if ((t & 31) == 0) s_max[t >> 5] = absmax;
    __syncthreads();
    absmax = s_max[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) absmax = fmaxf(absmax, s_max[i]);
    if (t * 8 >= K) return;   // (short rows: no division in warps that have no element)
    const float s = __fdiv_rn(absmax, 7.0f);
    if (t == 0) scale[r] = scale_out(absmax, s, role);
    store(AbsmaxCodes<T>(absmax, s));
  }
}

// Any even K, any alignment, any row length: two passes (the second one hits L2).
template <typename T, bool GIVEN>
__global__ void __launch_bounds__(256) quant_rowwise_generic_kernel(const T* __restrict__ x, int64_t K,
                                                                    int64_t ldx,
                                                                    const float* __restrict__ given_scale,
                                                                    uint8_t* __restrict__ packed,
                                                                    float* __restrict__ scale, int role) {
  __shared__ float s_max[8];
  const int64_t r = blockIdx.x;
  const T* src = x + r * ldx;
  const int t = threadIdx.x;
  float divisor, absmax = 0.f;
  if (GIVEN) {
    divisor = __ldg(given_scale + r);
  } else {
    for (int64_t k = t; k < K; k += 256) absmax = fmaxf(absmax, fabsf(to_f32(src[k])));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) absmax = fmaxf(absmax, __shfl_xor_sync(0xffffffffu, absmax, o));
    if ((t & 31) == 0) s_max[t >> 5] = absmax;
    __syncthreads();
    absmax = s_max[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) absmax = fmaxf(absmax, s_max[i]);
    divisor = __fdiv_rn(absmax, 7.0f);
    if (t == 0) scale[r] = scale_out(absmax, divisor, role);
  }
  const bool zero = !GIVEN && absmax == 0.f;
  uint8_t* dst = packed + r * (K / 2);
  for (int64_t i = t; i < K / 2; i += 256) {
    uint32_t lo = zero ? 0u : code4(to_f32(src[2 * i]), divisor);
    uint32_t hi = zero ? 0u : code4(to_f32(src[2 * i + 1]), divisor);
    dst[i] = (uint8_t)((hi << 4) | lo);
  }
}

// packed [n_words*4 bytes] -> int8, eight codes per thread-iteration.
__global__ void unpack_int4_kernel(const uint8_t* __restrict__ packed, int64_t n_bytes, int8_t* __restrict__ out) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t n_words = n_bytes / 4;
  const bool al = ((reinterpret_cast<uintptr_t>(packed) & 3) == 0) && ((reinterpret_cast<uintptr_t>(out) & 7) == 0);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_words; i += stride) {
    if (al) {
      const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(packed) + i);
      // byte b of w holds codes 2b (low nibble) and 2b+1 (high nibble)
      uint32_t o[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t acc = 0;
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const uint32_t byte = (w >> (8 * (2 * h + b))) & 0xFFu;
          const int lo = ((int)(byte << 28)) >> 28;
          const int hi = ((int)(byte << 24)) >> 28;
          acc |= ((uint32_t)lo & 0xFFu) << (16 * b);
          acc |= ((uint32_t)hi & 0xFFu) << (16 * b + 8);
        }
        o[h] = acc;
      }
      *reinterpret_cast<uint2*>(out + 8 * i) = make_uint2(o[0], o[1]);
    } else {
      for (int b = 0; b < 4; ++b) {
        const uint32_t byte = packed[4 * i + b];
        out[8 * i + 2 * b] = (int8_t)(((int)(byte << 28)) >> 28);
        out[8 * i + 2 * b + 1] = (int8_t)(((int)(byte << 24)) >> 28);
      }
    }
  }
  // tail bytes
  for (int64_t i = n_words * 4 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_bytes; i += stride) {
    const uint32_t byte = packed[i];
    out[2 * i] = (int8_t)(((int)(byte << 28)) >> 28);
    out[2 * i + 1] = (int8_t)(((int)(byte << 24)) >> 28);
  }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
template <typename T, int MODE, bool GIVEN>
static int launch_grouped_t(const T* x, int64_t rows, int64_t K, int64_t ldx, int gs, const int32_t* row_index,
                            int index_div, int64_t src_rows, const float* given, uint8_t* packed, float* scale, int role,
                            cudaStream_t st, const void* aux = nullptr, float eps = 0.f) {
  if (rows == 0 || K == 0) return I4TC_OK;
  // Enough blocks to fill the GPU several times over; beyond that a block walks several segments
  // of its rows so that loads of the next segment overlap the arithmetic of the current one.
  const int64_t row_blocks = (rows + quant_rows<MODE>() - 1) / quant_rows<MODE>();
  const int nseg = (int)((K + kQSeg - 1) / kQSeg);
  int spb = nseg;
  if (row_blocks < 2048) spb = (int)((int64_t)nseg * row_blocks / 2048);
  if (spb < 1) spb = 1;
  if (MODE == 3) spb = nseg;   // a warp normalises with the statistics of its whole row
  dim3 grid((unsigned)row_blocks, (unsigned)((nseg + spb - 1) / spb));
  I4TC_REQUIRE(grid.y <= 65535, I4TC_EINVAL, "K=%lld too large for the grouped quantiser", (long long)K);
#define I4TC_LAUNCH_G(LPG)                                                                             \
  I4TC_CUDA(launch_kernel(MODE >= 2, quant_grouped_kernel<T, LPG, MODE, GIVEN>, grid, quant_rows<MODE>() * 32, 0, st, x, rows, (int)K, \
                          ldx, row_index, index_div, src_rows, given, packed, scale, role, spb, static_cast<const T*>(aux), eps,     \
                          QuantOutMap{nullptr, nullptr, 0, 0, 0, 0, nullptr, 1, 0, 0}))
  switch (gs) {
    case 32: I4TC_LAUNCH_G(1); break;
    case 64: I4TC_LAUNCH_G(2); break;
    case 128: I4TC_LAUNCH_G(4); break;
    case 256: I4TC_LAUNCH_G(8); break;
    default: return fail(I4TC_EUNSUPPORTED, "group_size=%d not supported (32, 64, 128 or 256)", gs);
  }
#undef I4TC_LAUNCH_G
  I4TC_CUDA(cudaGetLastError());
  return I4TC_OK;
}

// Mapped-output launches (bf16 input, group size 128): MODE 1 = gather rows through row_index, MODE 2 = SwiGLU first.
template <int MODE>
static int launch_grouped_mapped(const __nv_bfloat16* x, int64_t rows, int64_t K, int64_t ldx, const int32_t* row_index,
                                 int index_div, int64_t src_rows, uint8_t* packed, float* scale, const QuantOutMap& out,
                                 cudaStream_t st) {
  if (rows == 0 || K == 0) return I4TC_OK;
  const int64_t row_blocks = (rows + kQRows - 1) / kQRows;
  const int nseg = (int)((K + kQSeg - 1) / kQSeg);
  int spb = nseg;
  if (row_blocks < 2048) spb = (int)((int64_t)nseg * row_blocks / 2048);
  if (spb < 1) spb = 1;
  dim3 grid((unsigned)row_blocks, (unsigned)((nseg + spb - 1) / spb));
  quant_grouped_kernel<__nv_bfloat16, 4, MODE, false, true><<<grid, 256, 0, st>>>(
      x, rows, (int)K, ldx, row_index, index_div, src_rows, nullptr, packed, scale, I4TC_ROLE_ACTIVATION, spb, nullptr, 0.f,
      out);
  I4TC_CUDA(cudaGetLastError());
  return I4TC_OK;
}

static int check_vec_input(const void* x, int dtype, int64_t ldx, const char* who) {
  const size_t es = dtype == I4TC_FP32 ? 4 : 2;
  I4TC_REQUIRE(aligned_to(x, 16) && (ldx * es) % 16 == 0, I4TC_EALIGN,
               "%s: input base and row stride must be 16-byte aligned", who);
  return I4TC_OK;
}

template <int MODE, bool GIVEN>
static int launch_grouped(const void* x, int dtype, int64_t rows, int64_t K, int64_t ldx, int64_t gs,
                          const int32_t* row_index, int index_div, const float* given, uint8_t* packed,
                          float* scale, int role, int device, void* stream, const void* aux = nullptr, float eps = 0.f,
                          int64_t src_rows = 0) {
  I4TC_REQUIRE(rows >= 0 && K >= 0 && gs > 0, I4TC_EINVAL, "negative size");
  I4TC_REQUIRE(gs % 2 == 0, I4TC_EINVAL, "group_size must be even");
  I4TC_REQUIRE(K % gs == 0, I4TC_EINVAL, "K must be divisible by group_size");
  I4TC_REQUIRE(K < (1ll << 31), I4TC_EINVAL, "K too large");
  I4TC_REQUIRE(role == I4TC_ROLE_ACTIVATION || role == I4TC_ROLE_WEIGHT, I4TC_EINVAL, "bad role");
  if (rows == 0 || K == 0) return I4TC_OK;
  I4TC_REQUIRE(x && packed && (GIVEN ? given != nullptr : scale != nullptr), I4TC_EINVAL, "null pointer");
  if (int rc = check_vec_input(x, dtype, ldx, "quant_grouped")) return rc;
  I4TC_REQUIRE(aligned_to(packed, 16), I4TC_EALIGN, "packed output must be 16-byte aligned");
  DeviceGuard guard(device);
  I4TC_CUDA(guard.err);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case I4TC_BF16:
      return launch_grouped_t<__nv_bfloat16, MODE, GIVEN>(static_cast<const __nv_bfloat16*>(x), rows, K, ldx,
                                                          (int)gs, row_index, index_div, src_rows, given, packed, scale,
                                                          role, st, aux, eps);
    case I4TC_FP16:
      if (MODE >= 2) break;
      return launch_grouped_t<__half, MODE >= 2 ? 0 : MODE, GIVEN>(static_cast<const __half*>(x), rows, K, ldx,
                                                                  (int)gs, row_index, index_div, src_rows, given, packed,
                                                                  scale, role, st);
    case I4TC_FP32:
      if (MODE >= 2) break;
      return launch_grouped_t<float, MODE >= 2 ? 0 : MODE, GIVEN>(static_cast<const float*>(x), rows, K, ldx,
                                                                 (int)gs, row_index, index_div, src_rows, given, packed,
                                                                 scale, role, st);
    default: break;
  }
  return fail(I4TC_EUNSUPPORTED, "unsupported input dtype %d", dtype);
}

template <typename T, bool GIVEN>
static int launch_rowwise_t(const T* x, int64_t rows, int64_t K, int64_t ldx, const float* given, uint8_t* packed,
                            float* scale, int role, cudaStream_t st) {
  const bool vec_ok = (K % 8 == 0) && K <= 16384 && aligned_to(x, 16) && (ldx * sizeof(T)) % 16 == 0 &&
                      aligned_to(packed, 4) && (K / 2) % 4 == 0;
  const unsigned grid = (unsigned)rows;
  if (!vec_ok) {
    quant_rowwise_generic_kernel<T, GIVEN><<<grid, 256, 0, st>>>(x, K, ldx, given, packed, scale, role);
  } else if (K <= 2048) {
    // A trigger in each of many short blocks costs more than a GEMM's early start gives: [8192, 128] 9.8 us with it, 7.3 without, [16384,
    // 1024] 18.4 and 13.9, [8192, 2048] 10.8 and 10.4; with the GEMM, [2048, 1024] x [1024, 1024] 11.4 and 11.6, [4096, 1024] x [1024,
    // 1024] 17.6 and 17.0.
    if (rows > 2048) quant_rowwise_kernel<T, 1, GIVEN, false><<<grid, 256, 0, st>>>(x, (int)K, ldx, given, packed, scale, role);
    else quant_rowwise_kernel<T, 1, GIVEN, true><<<grid, 256, 0, st>>>(x, (int)K, ldx, given, packed, scale, role);
  } else if (K <= 4096) {
    quant_rowwise_kernel<T, 2, GIVEN, true><<<grid, 256, 0, st>>>(x, (int)K, ldx, given, packed, scale, role);
  } else if (K <= 8192) {
    quant_rowwise_kernel<T, 4, GIVEN, true><<<grid, 256, 0, st>>>(x, (int)K, ldx, given, packed, scale, role);
  } else {
    quant_rowwise_kernel<T, 8, GIVEN, true><<<grid, 256, 0, st>>>(x, (int)K, ldx, given, packed, scale, role);
  }
  I4TC_CUDA(cudaGetLastError());
  return I4TC_OK;
}

template <bool GIVEN>
static int launch_rowwise(const void* x, int dtype, int64_t rows, int64_t K, int64_t ldx, const float* given,
                          uint8_t* packed, float* scale, int role, int device, void* stream) {
  I4TC_REQUIRE(rows >= 0 && K >= 0, I4TC_EINVAL, "negative size");
  I4TC_REQUIRE(K % 2 == 0, I4TC_EINVAL, "K must be even for INT4 packing");
  I4TC_REQUIRE(rows < (1ll << 31), I4TC_EINVAL, "too many rows");
  I4TC_REQUIRE(role == I4TC_ROLE_ACTIVATION || role == I4TC_ROLE_WEIGHT, I4TC_EINVAL, "bad role");
  if (rows == 0) return I4TC_OK;
  I4TC_REQUIRE(x || K == 0, I4TC_EINVAL, "null input");
  I4TC_REQUIRE((packed || K == 0) && (GIVEN ? given != nullptr : scale != nullptr), I4TC_EINVAL, "null pointer");
  DeviceGuard guard(device);
  I4TC_CUDA(guard.err);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case I4TC_BF16:
      return launch_rowwise_t<__nv_bfloat16, GIVEN>(static_cast<const __nv_bfloat16*>(x), rows, K, ldx, given,
                                                    packed, scale, role, st);
    case I4TC_FP16:
      return launch_rowwise_t<__half, GIVEN>(static_cast<const __half*>(x), rows, K, ldx, given, packed, scale,
                                             role, st);
    case I4TC_FP32:
      return launch_rowwise_t<float, GIVEN>(static_cast<const float*>(x), rows, K, ldx, given, packed, scale,
                                            role, st);
    default: break;
  }
  return fail(I4TC_EUNSUPPORTED, "unsupported input dtype %d", dtype);
}

}  // namespace i4tc

using namespace i4tc;

extern "C" int i4tc_quant_rowwise(const void* x, int dtype, int64_t rows, int64_t K, int64_t ldx, uint8_t* packed,
                                  float* scale, int role, int device, void* stream) {
  return launch_rowwise<false>(x, dtype, rows, K, ldx, nullptr, packed, scale, role, device, stream);
}

extern "C" int i4tc_quant_grouped(const void* x, int dtype, int64_t rows, int64_t K, int64_t ldx,
                                  int64_t group_size, uint8_t* packed, float* scale, int role, int device,
                                  void* stream) {
  return launch_grouped<0, false>(x, dtype, rows, K, ldx, group_size, nullptr, 1, nullptr, packed, scale, role,
                                  device, stream);
}

extern "C" int i4tc_quant_with_scales(const void* x, int dtype, int64_t rows, int64_t K, int64_t ldx,
                                      int64_t group_size, const float* scale, uint8_t* packed, int device,
                                      void* stream) {
  if (group_size == 0)
    return launch_rowwise<true>(x, dtype, rows, K, ldx, scale, packed, nullptr, I4TC_ROLE_ACTIVATION, device,
                                stream);
  return launch_grouped<0, true>(x, dtype, rows, K, ldx, group_size, nullptr, 1, scale, packed, nullptr,
                                 I4TC_ROLE_ACTIVATION, device, stream);
}

extern "C" int i4tc_moe_gather_quant(const void* x, int dtype, int64_t num_tokens, int64_t K, int64_t ldx,
                                     const int32_t* sorted_pairs, int64_t num_pairs, int64_t top_k, uint8_t* packed,
                                     float* scale, int device, void* stream) {
  I4TC_REQUIRE(top_k > 0 && top_k < (1 << 20), I4TC_EINVAL, "bad top_k");
  I4TC_REQUIRE(num_tokens >= 0, I4TC_EINVAL, "negative num_tokens");
  I4TC_REQUIRE(sorted_pairs || num_pairs == 0, I4TC_EINVAL, "null sorted_pairs");
  return launch_grouped<1, false>(x, dtype, num_pairs, K, ldx, 128, sorted_pairs, (int)top_k, nullptr, packed,
                                  scale, I4TC_ROLE_ACTIVATION, device, stream, nullptr, 0.f, num_tokens);
}

extern "C" int i4tc_moe_quant_fanout(const void* x, int64_t num_tokens, int64_t K, int64_t ldx, const int32_t* inv_pairs,
                                     int64_t top_k, int64_t num_rows, uint8_t* packed, float* scale, int device, void* stream) {
  I4TC_REQUIRE(top_k > 0 && top_k < (1 << 20) && num_tokens >= 0 && num_tokens * top_k < (1ll << 31), I4TC_EINVAL, "bad sizes");
  I4TC_REQUIRE(K > 0 && K % 128 == 0 && K < (1ll << 31) && num_rows >= 0, I4TC_EINVAL, "K must be a positive multiple of 128");
  if (num_tokens == 0 || num_rows == 0) return I4TC_OK;
  I4TC_REQUIRE(x && inv_pairs && packed && scale, I4TC_EINVAL, "null pointer");
  if (int rc = check_vec_input(x, I4TC_BF16, ldx, "moe_quant_fanout")) return rc;
  I4TC_REQUIRE(aligned_to(packed, 16), I4TC_EALIGN, "packed output must be 16-byte aligned");
  DeviceGuard guard(device);
  I4TC_CUDA(guard.err);
  const dim3 grid((unsigned)((num_tokens + kQRows - 1) / kQRows), (unsigned)((K + kQSeg - 1) / kQSeg));
  I4TC_REQUIRE(grid.y <= 65535, I4TC_EINVAL, "K=%lld too large", (long long)K);
  I4TC_CUDA(launch_kernel(true, quant_fanout_kernel, grid, 256, 0, static_cast<cudaStream_t>(stream),
                          static_cast<const __nv_bfloat16*>(x), num_tokens, (int)K, ldx, inv_pairs, (int)top_k, num_rows, packed, scale));
  return I4TC_OK;
}

extern "C" int i4tc_moe_ep_dispatch_quant(const void* x, int64_t num_tokens, int64_t K, int64_t ldx,
                                          const int32_t* sorted_pairs, int64_t num_pairs, int64_t top_k,
                                          const int32_t* slot, void* send_buf, int64_t row_bytes,
                                          const uint64_t* peer_bases, int64_t cap, int64_t my_rank, int device,
                                          void* stream) {
  I4TC_REQUIRE(top_k > 0 && top_k < (1 << 20) && num_tokens >= 0 && num_pairs >= 0, I4TC_EINVAL, "bad sizes");
  I4TC_REQUIRE(K > 0 && K % 128 == 0 && row_bytes == (K / 128) * 68, I4TC_EINVAL,
               "a row is 64 bytes of codes and one fp32 scale per 128 values");
  if (num_pairs == 0) return I4TC_OK;
  I4TC_REQUIRE(x && sorted_pairs && slot && (send_buf || peer_bases), I4TC_EINVAL, "null pointer");
  if (int rc = check_vec_input(x, I4TC_BF16, ldx, "moe_ep_dispatch_quant")) return rc;
  I4TC_REQUIRE(aligned_to(send_buf, 16), I4TC_EALIGN, "send buffer must be 16-byte aligned");
  I4TC_REQUIRE(peer_bases == nullptr || (cap > 0 && my_rank >= 0), I4TC_EINVAL, "peer destinations need cap and the rank");
  DeviceGuard guard(device);
  I4TC_CUDA(guard.err);
  const int64_t G = K / 128;
  QuantOutMap out;
  out.row_map = slot;
  out.rows_dev = nullptr;
  out.pk_gstride = 64;
  out.pk_rstride = row_bytes;
  out.sc_gstride = 1;
  out.sc_rstride = row_bytes / 4;
  out.dest_bases = reinterpret_cast<const unsigned long long*>(peer_bases);
  out.block_rows = (int)(1 + cap);
  out.my_block = (int)my_rank;
  out.scale_offset = G * 64;
  uint8_t* base = static_cast<uint8_t*>(send_buf);
  return launch_grouped_mapped<1>(static_cast<const __nv_bfloat16*>(x), num_pairs, K, ldx, sorted_pairs, (int)top_k,
                                  num_tokens, base, reinterpret_cast<float*>(base + G * 64), out,
                                  static_cast<cudaStream_t>(stream));
}

extern "C" int i4tc_moe_silu_mul_quant_rows(const void* h, int64_t max_rows, const int32_t* rows_dev, int64_t I,
                                            uint8_t* packed, float* scale, int device, void* stream) {
  I4TC_REQUIRE(max_rows >= 0 && I > 0 && I % 128 == 0, I4TC_EINVAL, "intermediate size must be a positive multiple of 128");
  if (max_rows == 0) return I4TC_OK;
  I4TC_REQUIRE(h && rows_dev && packed && scale, I4TC_EINVAL, "null pointer");
  if (int rc = check_vec_input(h, I4TC_BF16, 2 * I, "moe_silu_mul_quant_rows")) return rc;
  I4TC_REQUIRE(aligned_to(packed, 16), I4TC_EALIGN, "packed output must be 16-byte aligned");
  DeviceGuard guard(device);
  I4TC_CUDA(guard.err);
  QuantOutMap out;
  out.row_map = nullptr;
  out.rows_dev = rows_dev;
  out.pk_gstride = max_rows * 64;
  out.pk_rstride = 64;
  out.sc_gstride = max_rows;
  out.sc_rstride = 1;
  out.dest_bases = nullptr;
  out.block_rows = 1;
  out.my_block = 0;
  out.scale_offset = 0;
  return launch_grouped_mapped<2>(static_cast<const __nv_bfloat16*>(h), max_rows, I, 2 * I, nullptr, 1, 0, packed, scale,
                                  out, static_cast<cudaStream_t>(stream));
}

extern "C" int i4tc_moe_silu_mul_quant(const void* h, int64_t P, int64_t I, uint8_t* packed, float* scale,
                                       int device, void* stream) {
  return launch_grouped<2, false>(h, I4TC_BF16, P, I, 2 * I, 128, nullptr, 1, nullptr, packed, scale,
                                  I4TC_ROLE_ACTIVATION, device, stream);
}

extern "C" int i4tc_rmsnorm_quant_grouped(const void* x, int64_t rows, int64_t K, int64_t ldx, const void* norm_weight,
                                          float eps, int64_t group_size, uint8_t* packed, float* scale, int device,
                                          void* stream) {
  I4TC_REQUIRE(norm_weight != nullptr || rows == 0, I4TC_EINVAL, "null norm_weight");
  I4TC_REQUIRE(K % 32 == 0, I4TC_EINVAL, "K must be a multiple of 32");
  I4TC_REQUIRE(aligned_to(norm_weight, 16), I4TC_EALIGN, "norm_weight must be 16-byte aligned");
  I4TC_REQUIRE(eps >= 0.f, I4TC_EINVAL, "negative eps");
  return launch_grouped<3, false>(x, I4TC_BF16, rows, K, ldx, group_size, nullptr, 1, nullptr, packed, scale,
                                  I4TC_ROLE_ACTIVATION, device, stream, norm_weight, eps);
}

extern "C" int i4tc_unpack_int4_to_int8(const uint8_t* packed, int64_t rows, int64_t K, int8_t* out, int device,
                                        void* stream) {
  I4TC_REQUIRE(rows >= 0 && K >= 0 && K % 2 == 0, I4TC_EINVAL, "rows >= 0 and even K required");
  const int64_t n_bytes = rows * (K / 2);
  if (n_bytes == 0) return I4TC_OK;
  I4TC_REQUIRE(packed && out, I4TC_EINVAL, "null pointer");
  DeviceGuard guard(device);
  I4TC_CUDA(guard.err);
  const DeviceInfo* info;
  if (int rc = device_info(device, &info)) return rc;
  int64_t blocks = (n_bytes / 4 + 255) / 256;
  if (blocks < 1) blocks = 1;
  const int64_t cap = (int64_t)info->sm_count * 16;
  if (blocks > cap) blocks = cap;
  unpack_int4_kernel<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(packed, n_bytes, out);
  I4TC_CUDA(cudaGetLastError());
  return I4TC_OK;
}

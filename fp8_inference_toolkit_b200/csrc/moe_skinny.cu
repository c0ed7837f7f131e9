// Grouped W4A4 GEMM of a MoE layer with few rows per expert: weight streaming through register-fed tensor-core instructions.
//
// A decoding batch touches nearly every expert with a handful of rows, so the op is a stream of all experts' weights.  The tile
// kernel multiplies 128-row tiles (97 % padding at four rows) behind a chain of per-group hand-overs.  Here a warp owns 16
// weight rows of an expert and their whole K range; lane (g, t) holds 16 bytes of rows g and g + 8, which is an operand fragment once
// its nibbles are spread, so the weights go from HBM to registers (512 contiguous bytes per load, DEPTH groups ahead) and
// through nothing else.  A block's rows of the expert wait in shared memory as int8, at most TOK of them.  What hides the latency is the
// number of warps: no barrier, no shared-memory stage for the weights.
//
// The first TOK rows of every expert have block rows of their own; block rows past those look up what is left (find_pass), so that
// the rows of a popular expert run side by side and read its weights from the L2.  The host knows the mean only: there are as many
// extra block rows as one expert with all the rows would need, and most of them leave at once.
//
// One warp adds all K groups of its rows in ascending order with the tile kernel's operations (multiply by the row scale, fused
// multiply-add by the column scale), so the results are the tile kernel's bit for bit.  Nibble arithmetic and fragment
// layout as in skinny.cu.
//
// 128 experts of [1536, 2048] and [2048, 768] (321 MB of weights), top 8, both GEMMs behind a flushed L2, tile kernel -> this one,
// experts drawn uniformly: 64 tokens 181 -> 77 us (4.2 TB/s), 192 tokens 181 -> 101, 400 tokens 185 -> 149; with Zipf's weights 161 ->
// 81, 183 -> 118, 192 -> 185; all tokens on the same eight experts 58 -> 44, 61 -> 69, 85 -> 116.  (With a block taking an expert's
// passes one after the other: uniform 89, 108, 155; Zipf 103, 155, 206; eight experts 120, 142, 212; 1000 tokens on one expert 626, now
// 50.)  Bound by instructions and latency (the nibbles' 24 logic operations and four to sixteen products per warp and group), not by HBM:
// asking the L2 for a warp's whole K range beforehand changed nothing at 64 tokens and cost 20 % at 192.  Weights through shared memory
// (cp.async.bulk, two warps a block, ten warps an SM): 123 us at 64 tokens and 325 at 512.
#include "gemm.cuh"
#include "ptx.cuh"

namespace i4tc {

namespace {

constexpr int kMoeWarps = 8;

struct MoeSkinnyParams {
  const uint8_t* a;       // [G, P, 64]
  const float* sa;        // [G, P]
  const uint8_t* b;       // [E, G, N, 64]
  const float* sb;        // [E, G, N]
  const int32_t* offsets; // [E + 1]
  __nv_bfloat16* out;     // [P, N]
  long long P;
  int N, G;
  int E;                  // experts
};

__device__ __forceinline__ void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint4 low_nibbles(const uint4& w) {
  return make_uint4((w.x << 4) & 0xF0F0F0F0u, (w.y << 4) & 0xF0F0F0F0u, (w.z << 4) & 0xF0F0F0F0u, (w.w << 4) & 0xF0F0F0F0u);
}
__device__ __forceinline__ uint4 high_nibbles(const uint4& w) {
  return make_uint4(w.x & 0xF0F0F0F0u, w.y & 0xF0F0F0F0u, w.z & 0xF0F0F0F0u, w.w & 0xF0F0F0F0u);
}
__device__ __forceinline__ uint4 load_stream(const uint8_t* p) {   // read once: past L1
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// Shared memory: even codes [group][TOK][64 B] | odd codes [group][TOK][64 B] | row scales [group][TOK]
__host__ __device__ constexpr size_t moe_skinny_smem(int G, int tok) { return (size_t)G * tok * (128 + 4); }

// Where pass number `item` of those beyond every expert's first TOK rows begins: its expert and the row `first` of it.  False past
// the last pass.  Called by whole warps, which all come to the same answer: a lane counts the passes of a run of experts.
template <int TOK>
__device__ __forceinline__ bool find_pass(const int32_t* offsets, int E, int item, int& e, int& first) {
  const int lane = threadIdx.x & 31, run = (E + 31) / 32;
  const int x0 = min(E, lane * run), x1 = min(E, x0 + run);
  int mine = 0, prev = __ldg(offsets + x0);
#pragma unroll 4
  for (int x = x0; x < x1; ++x) {
    const int next = __ldg(offsets + x + 1);
    mine += max(next - prev - 1, 0) / TOK;
    prev = next;
  }
  if (__all_sync(0xffffffffu, mine == 0)) return false;
  int upto = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += v;
  }
  const unsigned found = __ballot_sync(0xffffffffu, upto > item);
  if (found == 0u) return false;
  const int l = __ffs(found) - 1;
  item -= __shfl_sync(0xffffffffu, upto - mine, l);
  for (e = l * run;; ++e) {   // (ends: the run holds the pass)
    const int n = max(__ldg(offsets + e + 1) - __ldg(offsets + e) - 1, 0) / TOK;
    if (item < n) break;
    item -= n;
  }
  first = (item + 1) * TOK;
  return true;
}

// NT: 8-row tiles of the expert's rows handled at once (TOK = 8 NT).  DEPTH: groups of weights in flight per warp.  BLOCKS: per SM.
template <int NT, int DEPTH, int BLOCKS>
__global__ void __launch_bounds__(kMoeWarps * 32, BLOCKS) moe_skinny_kernel(const MoeSkinnyParams p) {
  constexpr int TOK = 8 * NT;
  extern __shared__ __align__(128) uint8_t smem[];
  const int32_t* offsets = p.offsets;
  const uint8_t *pa = p.a, *pb = p.b;
  const float *psa = p.sa, *psb = p.sb;
  pdl_wait();
  pdl_fresh(offsets); pdl_fresh(pa); pdl_fresh(pb); pdl_fresh(psa); pdl_fresh(psb);
  pdl_trigger();
  // block row e < E: the first TOK rows of expert e; the block rows past them: what experts have beyond that
  int e = blockIdx.y, first = 0;
  if (e >= p.E && !find_pass<TOK>(offsets, p.E, e - p.E, e, first)) return;   // the whole block
  const int r0 = __ldg(offsets + e) + first, n = min(TOK, __ldg(offsets + e + 1) - r0);   // rows of this block
  if (n <= 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int n0 = (blockIdx.x * kMoeWarps + warp) * 16;
  const bool mine = n0 < p.N;   // a warp past the last rows only helps to stage
  const int G = p.G;
  uint8_t* lo_s = smem;
  uint8_t* hi_s = smem + (size_t)G * TOK * 64;
  float* sx_s = reinterpret_cast<float*>(smem + (size_t)G * TOK * 128);
  const long long row = (long long)e * G * p.N + (mine ? n0 : 0) + g;   // weight row of group 0
  const long long wstep = (long long)p.N * 64;

  uint4 wa[DEPTH], wb[DEPTH];
  float s0[DEPTH], s1[DEPTH];
  const uint8_t* wat = pb + row * 64 + t * 16;
  const float* sat = psb + row;
  auto fetch = [&](int d) {   // the groups in order
    wa[d] = load_stream(wat);
    wb[d] = load_stream(wat + 8 * 64);
    s0[d] = __ldg(sat);
    s1[d] = __ldg(sat + 8);
    wat += wstep;
    sat += p.N;
  };
#pragma unroll
  for (int d = 0; d < DEPTH; ++d)
    if (d < G) fetch(d);
  // ---- the block's rows (past the expert's end: zero codes, zero scales) ----
  for (int i = threadIdx.x; i < G * TOK * 4; i += kMoeWarps * 32) {
    const int j = i & 3, m = (i >> 2) % TOK, grp = (i >> 2) / TOK;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (m < n) v = __ldg(reinterpret_cast<const uint4*>(pa + ((long long)grp * p.P + r0 + m) * 64) + j);
    *reinterpret_cast<uint4*>(lo_s + (size_t)i * 16) = low_nibbles(v);
    *reinterpret_cast<uint4*>(hi_s + (size_t)i * 16) = high_nibbles(v);
  }
  for (int i = threadIdx.x; i < G * TOK; i += kMoeWarps * 32) {
    const int m = i % TOK, grp = i / TOK;
    sx_s[i] = m < n ? __ldg(psa + (long long)grp * p.P + r0 + m) * (1.0f / 256.0f) : 0.f;
  }
  __syncthreads();

  float f[NT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) f[nt][i] = 0.f;
  for (int base = 0; base < G; base += DEPTH) {
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) {
      const int grp = base + d;
      if (grp >= G) break;
      const uint4 alo = low_nibbles(wa[d]), ahi = high_nibbles(wa[d]), blo = low_nibbles(wb[d]), bhi = high_nibbles(wb[d]);
      const float sw0 = s0[d], sw1 = s1[d];
      if (grp + DEPTH < G) fetch(d);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int at = (grp * TOK + 8 * nt + g) * 64 + t * 16;
        const uint4 xlo = *reinterpret_cast<const uint4*>(lo_s + at), xhi = *reinterpret_cast<const uint4*>(hi_s + at);
        const float2 sx = *reinterpret_cast<const float2*>(sx_s + grp * TOK + 8 * nt + 2 * t);
        int c[4] = {0, 0, 0, 0};
        mma_s8(c, alo.x, blo.x, ahi.x, bhi.x, xlo.x, xhi.x);
        if (NT != 2) {   // two chains of two products (NT = 2 has no registers left for a second)
          int c2[4] = {0, 0, 0, 0};
          mma_s8(c2, alo.y, blo.y, ahi.y, bhi.y, xlo.y, xhi.y);
          mma_s8(c, alo.z, blo.z, ahi.z, bhi.z, xlo.z, xhi.z);
          mma_s8(c2, alo.w, blo.w, ahi.w, bhi.w, xlo.w, xhi.w);
#pragma unroll
          for (int i = 0; i < 4; ++i) c[i] += c2[i];
        } else {
          mma_s8(c, alo.y, blo.y, ahi.y, bhi.y, xlo.y, xhi.y);
          mma_s8(c, alo.z, blo.z, ahi.z, bhi.z, xlo.z, xhi.z);
          mma_s8(c, alo.w, blo.w, ahi.w, bhi.w, xlo.w, xhi.w);
        }
        // (acc * scale_a[g, m]) * scale_b[g, n]; 2^-8 rides on the row's scale (exact)
        f[nt][0] = fmaf(__int2float_rn(c[0]) * sx.x, sw0, f[nt][0]);
        f[nt][1] = fmaf(__int2float_rn(c[1]) * sx.y, sw0, f[nt][1]);
        f[nt][2] = fmaf(__int2float_rn(c[2]) * sx.x, sw1, f[nt][2]);
        f[nt][3] = fmaf(__int2float_rn(c[3]) * sx.y, sw1, f[nt][3]);
      }
    }
  }

  // ---- lanes g and g ^ 1 swap a row each, so that a lane stores pairs of columns: n0 + (g & ~1) + {0, 1} (+ 8) ----
  const bool odd = (g & 1) != 0;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const float o0 = __shfl_xor_sync(0xffffffffu, odd ? f[nt][0] : f[nt][1], 4);
    const float o1 = __shfl_xor_sync(0xffffffffu, odd ? f[nt][2] : f[nt][3], 4);
    const int m = 8 * nt + 2 * t + (odd ? 1 : 0);
    if (m < n && mine) {
      __nv_bfloat16* dst = p.out + (long long)(r0 + m) * p.N + n0 + (g & ~1);
      const __nv_bfloat162 lo = odd ? __floats2bfloat162_rn(o0, f[nt][1]) : __floats2bfloat162_rn(f[nt][0], o0);
      const __nv_bfloat162 hi = odd ? __floats2bfloat162_rn(o1, f[nt][3]) : __floats2bfloat162_rn(f[nt][2], o1);
      *reinterpret_cast<__nv_bfloat162*>(dst) = lo;
      *reinterpret_cast<__nv_bfloat162*>(dst + 8) = hi;
    }
  }
}

constexpr size_t kMoeSkinnyMaxSmem = 110 * 1024;

template <int NT, int DEPTH, int BLOCKS>
int launch_nt(const MoeSkinnyParams& p, cudaStream_t st) {
  // The limit belongs to the function, not to a launch, so it is the most that moe_skinny_applicable admits: with each call's own
  // size, a thread with fewer groups could lower it between another thread's setting and its launch.
  static bool configured[64] = {false};
  int dev = 0;
  I4TC_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !configured[dev]) {
    I4TC_CUDA(cudaFuncSetAttribute(moe_skinny_kernel<NT, DEPTH, BLOCKS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kMoeSkinnyMaxSmem));
    if (dev < 64) configured[dev] = true;
  }
  const size_t smem = moe_skinny_smem(p.G, 8 * NT);
  const int blocks = (p.N + 16 * kMoeWarps - 1) / (16 * kMoeWarps);
  // passes beyond the experts' first: at most (P - 1) / TOK, when every row goes to one expert
  const unsigned rows = (unsigned)(p.E + (p.P - 1) / (8 * NT));
  I4TC_CUDA(launch_kernel(true, moe_skinny_kernel<NT, DEPTH, BLOCKS>, dim3((unsigned)blocks, rows), kMoeWarps * 32, smem, st, p));
  return I4TC_OK;
}

}  // namespace

// 8-row tiles handled at once: the rows an expert has on average, with room for most of their spread.  Beyond 26 rows an expert
// the tile kernel takes over: it needs 185 us from 4 to 64 rows an expert, this kernel 149 at 25 (uniform; Zipf 185), and 195 with eight
// tiles at 44.  What the line costs: from 12 rows an expert on, calls whose rows all go to a few experts are slower than with tiles (by
// 1.1 to 1.5, figures above), which the host cannot tell from the mean.  Handing experts with more than 32 or 64 rows to the
// tile kernel in a launch of its own made mixed loads slower (Zipf at 300 tokens 179 -> 209) and was not kept.
static int nt_for(long long num_pairs, long long num_experts) {
  return num_pairs <= 5 * num_experts ? 1 : num_pairs <= 12 * num_experts ? 2 : 4;
}

bool moe_skinny_applicable(long long num_pairs, long long N, int G, long long num_experts) {
  return num_pairs <= 26 * num_experts && N % 16 == 0 && num_experts <= 32768 &&
         moe_skinny_smem(G, 8 * nt_for(num_pairs, num_experts)) <= kMoeSkinnyMaxSmem;
}

int launch_moe_skinny(const uint8_t* a, const float* sa, const uint8_t* b, const float* sb, const int32_t* offsets, void* out,
                      long long P, long long N, int G, long long num_experts, cudaStream_t st) {
  MoeSkinnyParams p;
  p.a = a; p.sa = sa; p.b = b; p.sb = sb; p.offsets = offsets;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.P = P; p.N = (int)N; p.G = G; p.E = (int)num_experts;
  switch (nt_for(P, num_experts)) {
    case 1: return launch_nt<1, 2, 4>(p, st);
    case 2: return launch_nt<2, 3, 3>(p, st);
    default: return launch_nt<4, 2, 2>(p, st);
  }
}

}  // namespace i4tc

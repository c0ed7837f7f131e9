// Device helpers shared by the tcgen05 tile kernels: bounded mbarrier waits, operand descriptors, the column order of
// the accumulator tiles, output conversion and the ragged stores.
#pragma once
#include "gemm.cuh"
#include "ptx.cuh"

namespace i4tc {

using namespace ptx;

constexpr int kBM = 128;             // rows of the P tile == TMEM lanes
constexpr int kI8Row = 128;          // bytes of one 8-bit row of one group (the swizzle width)
constexpr uint64_t kWaitLimitNs = 2000000000ull;  // 2 s

struct TileInfo {
  int p0, q0;        // first row of the P / Q tile
  int p_lim, q_lim;  // exclusive row limits for output
  int zq;            // slab offset of the Q operand (MoE: expert * G)
  long long sq_off;  // float offset into sq (MoE: expert * sq_estride)
  int g0, g1;        // K groups [g0, g1) of this work item (all of them unless split-K)
  int split;
};

// Static persistent schedule: CTA b takes tiles b, b + grid, ...  P tiles vary fastest so that
// CTAs running together share Q (weight) tiles in L2.
// With CG = 2 a work item is a 256-row P tile of a CTA pair; rank r of the pair owns rows 128 r .. 128 r + 127
// of it (p.num_p_tiles then counts 256-row tiles).
template <int CG = 1>
struct SchedT {
  int tile;
  int e;
  int tile_base;
  int rank;
  __device__ SchedT() : tile(blockIdx.x / CG), e(0), tile_base(0), rank(CG == 2 ? (int)cluster_ctarank() : 0) {}
  template <int BN>
  __device__ bool next(const GemmParams& p, TileInfo& ti) {
    if (p.expert_offsets == nullptr) {
      const int per_split = p.num_p_tiles * p.num_q_tiles;
      if (tile >= per_split * p.splits) return false;
      const int sp = tile / per_split, local = tile - sp * per_split;
      const int pt = local % p.num_p_tiles, qt = local / p.num_p_tiles;
      ti.p0 = pt * (kBM * CG) + rank * kBM; ti.q0 = qt * BN; ti.p_lim = p.P_rows; ti.q_lim = p.Q_rows; ti.zq = 0; ti.sq_off = 0;
      ti.split = sp; ti.g0 = sp * p.groups_per_split;
      ti.g1 = min(p.G, ti.g0 + p.groups_per_split);
    } else {
      for (;;) {
        if (e >= p.num_experts) return false;
        const int r0 = __ldg(p.expert_offsets + e), r1 = __ldg(p.expert_offsets + e + 1);
        const int npt = (r1 - r0 + kBM - 1) / kBM;
        const int nt = npt * p.num_q_tiles;
        if (tile < tile_base + nt) {
          const int local = tile - tile_base;
          const int pt = local % npt, qt = local / npt;
          ti.p0 = r0 + pt * kBM; ti.p_lim = r1; ti.q0 = qt * BN; ti.q_lim = p.Q_rows;
          ti.zq = e * p.G; ti.sq_off = (long long)e * p.sq_estride;
          ti.split = 0; ti.g0 = 0; ti.g1 = p.G;
          break;
        }
        tile_base += nt; ++e;
      }
    }
    tile += gridDim.x / CG;
    return true;
  }
};
// Bounded mbarrier wait, uniform across the warp.  Returns false (and raises the abort flag)
// when the limit expires or another role has already aborted.  The common case -- the phase has
// already completed -- is one non-blocking probe; everything else is the rare path.
__device__ __forceinline__ bool wait_bar_slow(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  bool ok = mbar_try_wait(bar, parity);
  if (!ok) {
    const uint64_t t0 = globaltimer_ns();
    uint32_t spins = 0;
    for (;;) {
      ok = mbar_try_wait(bar, parity);
      if (ok) break;
      if ((++spins & 63u) == 0) {
        if (*abort_flag) break;
        if (globaltimer_ns() - t0 > kWaitLimitNs) break;
      }
    }
  }
  ok = __all_sync(0xffffffffu, ok);
  if (!ok) *abort_flag = 1;
  return ok;
}
// The same wait for a role that runs as a single thread (no warp vote).
__device__ __forceinline__ bool wait_bar_thread(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_test_wait(bar, parity)) return true;
  bool ok = mbar_try_wait(bar, parity);
  if (!ok) {
    const uint64_t t0 = globaltimer_ns();
    uint32_t spins = 0;
    for (;;) {
      ok = mbar_try_wait(bar, parity);
      if (ok) break;
      if ((++spins & 63u) == 0) {
        if (*abort_flag) break;
        if (globaltimer_ns() - t0 > kWaitLimitNs) break;
      }
    }
  }
  if (!ok) *abort_flag = 1;
  return ok;
}
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (__all_sync(0xffffffffu, mbar_test_wait(bar, parity))) return true;
  return wait_bar_slow(bar, parity, abort_flag);
}

// Arrival on a barrier that, for CG = 2, may live in the peer CTA (`bar` is then a shared::cluster address).
template <int CG>
__device__ __forceinline__ void arrive_bar(uint32_t bar) {
  if (CG == 2) mbar_arrive_cluster(bar);
  else mbar_arrive(bar);
}

__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
  // K-major, 128-byte swizzle: rows 128 B apart, 8-row groups 1024 B apart (SBO), LBO unused (1),
  // descriptor version 1 (sm_100), layout type 2 (SWIZZLE_128B).
  uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Row order of a converted Q tile.  After tcgen05.ld.16x256b a lane (lr, lq) holds, of every 32-column chunk, the column
// pairs 8 kk + 2 lq + {0, 1}, kk = 0..3.  The converters therefore store Q row n of a 32-row block at row
// qperm(n) = 8 * ((n >> 1) & 3) + 2 * (n >> 3) + (n & 1): accumulator column 8 kk + 2 lq + e is then output column
// 8 lq + 2 kk + e, a lane's four pairs are eight CONSECUTIVE output columns, and a chunk row leaves as one 16-byte store
// per lane with no exchange between lanes (a 4 x 4 transpose in the quad costs 4 shuffles and 16 selects per chunk row).
// The map is its own inverse.  Tiles that reach shared memory without the converters (int8 operands) keep the
// natural order (QP = false below).
__host__ __device__ constexpr int qperm(int n) {
  return (n & ~31) | (((n >> 1) & 3) << 3) | (((n >> 3) & 3) << 1) | (n & 1);
}
// first of the two output columns (inside a 32-column chunk) of a lane's pair kk
template <bool QP>
__device__ __forceinline__ constexpr int pair_col(int kk, int lq) { return QP ? lq * 8 + kk * 2 : kk * 8 + lq * 2; }

template <typename OutT>
__device__ __forceinline__ OutT cast_out(float v);
template <>
__device__ __forceinline__ __nv_bfloat16 cast_out<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half cast_out<__half>(float v) { return __float2half_rn(v); }

template <typename OutT>
__device__ __forceinline__ uint32_t pack_pair(float2 v) {
  union { OutT h[2]; uint32_t u; } pk;
  pk.h[0] = cast_out<OutT>(v.x); pk.h[1] = cast_out<OutT>(v.y);
  return pk.u;
}

// Writes the column pair (q, q + 1) of tile row prow without any alignment assumption beyond what
// `pair_ok` promises (even ldc, 4-byte aligned base): 16-bit output, normal or swapped orientation.
template <typename OutT, bool SWAP>
__device__ __forceinline__ void store_pair(OutT* out, long long ldc, int prow, int q, int q_lim, float2 v, bool pair_ok) {
  if (!SWAP) {
    OutT* dst = out + (long long)prow * ldc + q;
    if (q + 1 < q_lim && pair_ok) {
      *reinterpret_cast<uint32_t*>(dst) = pack_pair<OutT>(v);
    } else {
      if (q < q_lim) dst[0] = cast_out<OutT>(v.x);
      if (q + 1 < q_lim) dst[1] = cast_out<OutT>(v.y);
    }
  } else {
    if (q < q_lim) out[(long long)q * ldc + prow] = cast_out<OutT>(v.x);
    if (q + 1 < q_lim) out[(long long)(q + 1) * ldc + prow] = cast_out<OutT>(v.y);
  }
}

}  // namespace i4tc

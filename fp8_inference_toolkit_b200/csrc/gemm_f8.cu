// Per-group W4A4 GEMM for large M on SM pairs: operands expanded to e4m3 beforehand, fp32 accumulators.
//
// What bounds the converting kernel (gemm_kernel.cu) with a flush per K group is the drain: an int32 -> fp32 conversion,
// a multiply and a multiply-add per accumulator, next to converter warps and their shared-memory traffic (96 KB per
// group tile of 128 x 256).  Every code of -8..7 is an e4m3 number and a group's sum is at most 2^13 (128 products of 64), so
// tcgen05.mma kind::f8f6f4 gives the same integers as exact fp32 values at the same rate: no conversion in the drain.
// The codes are expanded once per call (expand_e4m3_kernel: 1.5 bytes of traffic per code) instead of once per tile, TMA
// writes the swizzled operand tiles itself, and the warps that converted drain instead.  Results are bit-identical.
//   [8192, 4096] x [24576, 4096]: 1282 -> 869 us (expansion included); with the zero-point term 1900 -> 1150 us
//   [4096, 12288] x [4096, 12288]: 360 -> 262 us;  [1000, 4096] x [6144, 4096]: 60 -> 51 us
// A group tile of 256 x 256 takes a pair about 1110 cycles: the tensor cores need 512 of them, the packed fp32 arithmetic
// 570 (640 next to MMAs).  Timed on one SM without barriers, the drain of a 128 x 256 tile takes 690-740 cycles alone and 980-1020
// next to MMAs, whether by 8 or 16 warps and with one or two TMEM loads in flight: 80 LDS.128 of scales take 150 cycles
// alone and 580 next to MMAs, whose operand reads go first, and TMEM loads (270) are not slowed.  Knocked out one by one: the arithmetic
// 80 us of 322 ([8192, 4096] x [8192, 4096]), the multiplies 20, the output stores 16.  Measured and not kept: two MMA-issuing warps,
// on alternate groups or on the halves of a tile with an accumulator each (+0-8 %), 160-column tiles with three accumulators
// (+19 %), TMEM loads a step ahead across groups (+5-10 %), scales a group ahead in registers (+30 %), pairs packed by
// explicit 64-bit registers (+4 %), row scales doubled in shared memory (+2 %).
//
// Roles (12 warps): warp 0 TMA producer, warp 1 MMA issuer (leader) or reporter (second CTA), warps 2-3 scale
// loaders, the others epilogue.  Every wait is bounded as in gemm_kernel.cu.
#include "gemm_dev.cuh"

namespace i4tc {

using namespace ptx;

constexpr int kF8EpiWarp0 = 4;   // warps 0..3: TMA producer, MMA issuer, two scale loaders

// Four consecutive floats of shared memory as two pairs.
__device__ __forceinline__ void lds_pairs(uint32_t addr, float2& a, float2& b) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a.x), "=f"(a.y), "=f"(b.x), "=f"(b.y) : "r"(addr));
}

template <int BN>
struct F8Cfg {
  static constexpr int NT = BN > 128 ? 2 : 4;             // accumulators in the 512 TMEM columns
  // 8 epilogue warps, 32 rows x BN / 2 columns of every accumulator each: what a warp pays per group (probes, arrivals, row
  // scales, index arithmetic) is spread over 64 to 128 columns.  Against BN / 16 warps of 64 columns, [8192, 4096] x
  // [24576, 4096]: 981 -> 869 us at 256, 983 -> 924 at 192, 985 -> 928 at 128 columns
  static constexpr int EW = 8;
  static constexpr int CW = BN / 2;
  static constexpr int STEP = BN == 192 ? 16 : 32;        // columns per TMEM load (the other one: 2 to 4 % slower)
  // registers per thread of warps 0..3 and of the epilogue, within what the launch allocates (384 threads x 168):
  // 128 * 56 + 256 * 224, CW of the latter for the running sums
  static constexpr int REG_LOW = 56, REG_EPI = 224;
  static constexpr int THREADS = (kF8EpiWarp0 + EW) * 32;
  static constexpr int QR = BN / 2;                       // Q rows staged by each CTA of the pair
  static constexpr int ST_P = kBM * kI8Row, ST_Q = QR * kI8Row;
  static constexpr int NS = BN > 128 ? 6 : 8;             // stages: operand tiles and scales of one K group
  static_assert(NS >= NT, "the epilogue waits on the barrier ring of the stages");
  // floats per scale stage: row scales, column scales; then the rows' zero points (each twice, as a pair) and the columns' sums
  static constexpr int SC_Z = kBM + BN, SC_F = SC_Z + 2 * kBM + BN;
  static constexpr int OFF_SC = NS * (ST_P + ST_Q);
  static constexpr int OFF_BAR = OFF_SC + NS * SC_F * 4;
  static constexpr int NUM_BARS = 3 * NS + NT;
  static constexpr int OFF_MISC = OFF_BAR + NUM_BARS * 8;
  static constexpr int SMEM_BYTES = OFF_MISC + 16 + 1024;
};

template <int BN, bool AZP>
__global__ void __launch_bounds__(F8Cfg<BN>::THREADS, 1)
w4a4_group_f8_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ CUtensorMap tmP,
                     const __grid_constant__ CUtensorMap tmQ, const int p_pitch, const int q_pitch) {
  using C = F8Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;

  // full: this CTA's operand tiles (1 arrival + bytes) and scales (32 lanes) of the stage have landed; in the leader also
  // the peer's (1 arrival).  done: the MMAs that read the stage are complete -- "stage free" and "accumulator full".
  const uint32_t bar_full = sbase + C::OFF_BAR;
  const uint32_t bar_done = bar_full + C::NS * 8;
  const uint32_t bar_sc_empty = bar_done + C::NS * 8;   // this CTA's epilogue warps have read the stage's scales
  const uint32_t bar_tm = bar_sc_empty + C::NS * 8;      // leader: both CTAs have drained the accumulator
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::OFF_MISC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + C::OFF_MISC + 8);

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::NS; ++i) {
      mbar_init(bar_full + i * 8, leader ? 34 : 33); mbar_init(bar_done + i * 8, 1); mbar_init(bar_sc_empty + i * 8, C::EW);
    }
    for (int i = 0; i < C::NT; ++i) mbar_init(bar_tm + i * 8, C::EW * 2);
    *abort_flag = 0;
    fence_mbar_init();
    prefetch_tensormap(&tmP);
    prefetch_tensormap(&tmQ);
  }
  if (warp == 1) { tmem_alloc_cg2(smem_u32(tmem_slot), 512); tmem_relinquish_cg2(); }
  pdl_wait();   // the expanded operands, the scales and the output
  tc_fence_before_sync();
  cluster_sync();   // the peer's barriers are initialised before anything arrives on them
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < 4) {
    setmaxnreg_dec<C::REG_LOW>();
    SchedT<2> sched;
    TileInfo ti;
    uint32_t it = 0;
    bool ok = true;
    if (warp == 0) {
      // ---------------- TMA producer: group g of an operand starts at row g * pitch of its expanded form ----------------
      while (ok && sched.template next<BN>(p, ti)) {
        for (int g = ti.g0; g < ti.g1; ++g, ++it) {
          const uint32_t s = it % C::NS, ph = (it / C::NS) & 1u;
          ok = wait_bar(bar_done + s * 8, ph ^ 1u, abort_flag);
          if (!ok) break;
          if (lane == 0) {
            const uint32_t full = bar_full + s * 8;
            const uint32_t dst = sbase + s * (C::ST_P + C::ST_Q);
            mbar_arrive_expect_tx(full, C::ST_P + C::ST_Q);
            tma_load_2d(dst, &tmP, full, 0, g * p_pitch + ti.p0);
            tma_load_2d(dst + C::ST_P, &tmQ, full, 0, g * q_pitch + ti.q0 + (int)rank * C::QR);
          }
          __syncwarp();
        }
      }
      if (!ok) {
        // aborting: wait (bounded) for copies that may still be in flight into this CTA's shared memory
        const uint32_t n = it < (uint32_t)C::NS ? it : (uint32_t)C::NS;
        for (uint32_t j = it - n; j < it; ++j) {
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try_wait(bar_full + (j % C::NS) * 8, (j / C::NS) & 1u)) {
            if (globaltimer_ns() - t0 > 100000000ull) break;
          }
        }
      }
    } else if (warp == 1) {
      if (leader) {
        // ---------------- MMA issuer ----------------
        // (elect.sync, not lane == 0: timed, an MMA costs the thread 41 cycles instead of 85)
        if (elect_one()) {
          // D = fp32 (1 << 4), A = B = e4m3 (0), K-major, N >> 3 at bit 17, M >> 4 at bit 24
          constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((kBM * 2) >> 4) << 24);
          bool ready = false;
          while (ok && sched.template next<BN>(p, ti)) {
            for (int g = ti.g0; g < ti.g1; ++g, ++it) {
              const uint32_t s = it % C::NS, buf = it % C::NT;
              if (!ready) {
                ok = wait_bar_thread(bar_full + s * 8, (it / C::NS) & 1u, abort_flag) &&
                     wait_bar_thread(bar_tm + buf * 8, ((it / C::NT) & 1u) ^ 1u, abort_flag);
                if (!ok) break;
              }
              tc_fence_after_sync();
              // the next group's probes are in flight under this group's MMAs (an index past the end is never waited for)
              ready = mbar_test_wait(bar_full + ((it + 1) % C::NS) * 8, ((it + 1) / C::NS) & 1u) &
                      mbar_test_wait(bar_tm + ((it + 1) % C::NT) * 8, (((it + 1) / C::NT) & 1u) ^ 1u);
              const uint32_t aP = sbase + s * (C::ST_P + C::ST_Q);
              const uint64_t dP = make_desc(aP), dQ = make_desc(aP + C::ST_P);
#pragma unroll
              for (int k = 0; k < 4; ++k)
                mma_f8_cg2(tmem_base + buf * BN, dP + (uint64_t)(2 * k), dQ + (uint64_t)(2 * k), idesc, k == 0 ? 0u : 1u);
              tc_commit_cg2_both(bar_done + s * 8, (uint16_t)3);   // one arrival in each CTA
            }
          }
        }
      } else {
        // ---------------- second CTA: report to the leader that a group's stage and scales are here ----------------
        const uint32_t arr_peer = mapa_shared(bar_full, 0);
        while (ok && sched.template next<BN>(p, ti)) {
          for (int g = ti.g0; g < ti.g1; ++g, ++it) {
            ok = wait_bar(bar_full + (it % C::NS) * 8, (it / C::NS) & 1u, abort_flag);
            if (!ok) break;
            if (lane == 0) mbar_arrive_cluster(arr_peer + (it % C::NS) * 8);
            __syncwarp();
          }
        }
      }
      __syncwarp();   // the issuing thread rejoins its warp before the block-wide teardown
    } else {
      // ---------------- scale loaders (warps 2 and 3 take alternate K groups) ----------------
      // row scales are stored so that a lane's four rows (8 a + lr) are four consecutive floats
      const int rslot = (lane & 7) * 4 + (lane >> 3);
      while (ok && sched.template next<BN>(p, ti)) {
        for (int g = ti.g0; g < ti.g1; ++g, ++it) {
          if ((it & 1u) != (uint32_t)(warp - 2)) continue;
          const uint32_t ss = it % C::NS;
          ok = wait_bar(bar_sc_empty + ss * 8, ((it / C::NS) & 1u) ^ 1u, abort_flag);
          if (!ok) break;
          const uint32_t dst = sbase + C::OFF_SC + ss * (C::SC_F * 4);
#pragma unroll
          for (int j = 0; j < kBM / 32; ++j) {
            const int row = ti.p0 + j * 32 + lane;
            const bool v = row < ti.p_lim;
            cp_async_4_zfill(dst + (uint32_t)(j * 32 + rslot) * 4u, v ? p.sp + (long long)g * p.sp_gstride + row : p.sp, v);
            if (AZP) {
              // row 8 a + lr of the 32 at [a / 2][lr][a & 1], so that one 16-byte load gives a lane the pairs of two of its rows
              const uint32_t at = dst + (uint32_t)(C::SC_Z + j * 64 + ((lane >> 4) * 8 + (lane & 7)) * 4 + ((lane >> 3) & 1) * 2) * 4u;
              const float* src = v ? p.zp + (long long)g * p.sp_gstride + row : p.sp;
              cp_async_4_zfill(at, src, v);
              cp_async_4_zfill(at + 4, src, v);
            }
          }
#pragma unroll
          for (int j = 0; j < BN / 32; ++j) {
            const int q = ti.q0 + j * 32 + lane;
            const bool v = q < ti.q_lim;
            cp_async_4_zfill(dst + (uint32_t)(kBM + j * 32 + lane) * 4u, v ? p.sq + (long long)g * p.sq_gstride + q : p.sq, v);
            if (AZP) cp_async_4_zfill(dst + (uint32_t)(C::SC_Z + 2 * kBM + j * 32 + lane) * 4u, v ? p.zq + (long long)g * p.sq_gstride + q : p.sq, v);
          }
          cp_async_mbar_arrive_noinc(bar_full + ss * 8);   // fires when this lane's copies have landed
        }
      }
      cp_async_wait_all();   // nothing of this warp is in flight into shared memory at teardown
    }
  } else {
    // ---------------- epilogue: 32 rows x CW columns of every accumulator per warp ----------------
    setmaxnreg_inc<C::REG_EPI>();
    constexpr int CW = C::CW, NCH = CW / 32, STEP = C::STEP;
    const int quad = warp & 3, col_base = ((warp - kF8EpiWarp0) >> 2) * CW;
    const int lq = lane & 3, lr = lane >> 2;
    const uint32_t arr_tm = mapa_shared(bar_tm, 0);
    const uint32_t tm_warp = tmem_base + ((uint32_t)(quad * 32) << 16) + col_base;
    const uint32_t sc_row = sbase + C::OFF_SC + (uint32_t)(quad * 32 + lr * 4) * 4u;
    const uint32_t sc_col = sbase + C::OFF_SC + (uint32_t)(kBM + col_base + lq * 8) * 4u;
    const uint32_t z_row = sbase + C::OFF_SC + (uint32_t)(C::SC_Z + quad * 64 + lr * 4) * 4u;
    constexpr uint32_t Z_COL = (uint32_t)(C::SC_Z + kBM) * 4u;   // from a column's scale to its sum
    SchedT<2> sched;
    TileInfo ti;
    uint32_t it = 0, s = 0, ph = 0, buf = 0;   // group, its stage, the stage's phase, its accumulator
    bool ok = true, pre = false;   // pre: the next group was seen complete under this one's arithmetic
    __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.out);
    while (sched.template next<BN>(p, ti)) {
      float2 f[CW / 2];   // [a][c][kk]: row 8a + lr, columns c * 32 + 8 lq + 2 kk + {0, 1}
#pragma unroll
      for (int i = 0; i < CW / 2; ++i) f[i] = make_float2(0.f, 0.f);
      for (int g = ti.g0; g < ti.g1; ++g) {
        const uint32_t st = s * (C::SC_F * 4);
        // (the scales of the group arrived with its operands)
        if (!__all_sync(0xffffffffu, pre)) ok = wait_bar(bar_done + s * 8, ph, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
        float2 sp[4], zp[AZP ? 4 : 1];
        {
          float2 a, b;
          lds_pairs(sc_row + st, a, b);
          sp[0] = make_float2(a.x, a.x); sp[1] = make_float2(a.y, a.y); sp[2] = make_float2(b.x, b.x); sp[3] = make_float2(b.y, b.y);
        }
        if constexpr (AZP) { lds_pairs(z_row + st, zp[0], zp[1]); lds_pairs(z_row + st + 128, zp[2], zp[3]); }
#pragma unroll
        for (int u = 0; u < CW / STEP; ++u) {   // STEP columns at a time: a 32-column chunk c, or half of one from pair kk0 on
          const int c = u * STEP / 32, kk0 = (u * STEP / 8) & 3;
          uint32_t r[2][STEP / 2];
          const uint32_t tm = tm_warp + buf * BN + u * STEP;
          if constexpr (STEP == 32) {
            tmem_ld_16x256b_x4(tm, r[0]);
            tmem_ld_16x256b_x4(tm + (16u << 16), r[1]);
          } else {
            tmem_ld_16x256b_x2(tm, r[0]);
            tmem_ld_16x256b_x2(tm + (16u << 16), r[1]);
          }
          float2 sq[STEP / 8], zq[AZP ? STEP / 8 : 1];
#pragma unroll
          for (int i = 0; i < STEP / 8; i += 2) {
            const uint32_t at = sc_col + st + (uint32_t)(c * 32 + kk0 * 2 + i * 2) * 4u;
            lds_pairs(at, sq[i], sq[i + 1]);
            if constexpr (AZP) lds_pairs(at + Z_COL, zq[i], zq[i + 1]);
          }
          tmem_ld_wait();
          if (u == CW / STEP - 1) {
            // all of this warp's part of the accumulator and of the scales is in registers: hand both back
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) { mbar_arrive_cluster(arr_tm + buf * 8); mbar_arrive(bar_sc_empty + s * 8); }
            pre = mbar_test_wait(bar_done + ((it + 1) % C::NS) * 8, ((it + 1) / C::NS) & 1u);
          }
          auto fold = [&](int a, int kk) {
            const int i = 4 * kk + 2 * (a & 1);
            float2 d = make_float2(__uint_as_float(r[a >> 1][i]), __uint_as_float(r[a >> 1][i + 1]));
            if constexpr (AZP) d = __ffma2_rn(zp[a], zq[kk], d);
            float2& acc = f[(a * NCH + c) * 4 + kk0 + kk];
            acc = __ffma2_rn(__fmul2_rn(d, sp[a]), sq[kk], acc);
          };
          if constexpr (STEP == 32) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) { fold(0, kk); fold(1, kk); fold(2, kk); fold(3, kk); }
          } else {
#pragma unroll
            for (int a = 0; a < 4; ++a) { fold(a, 0); fold(a, 1); }
          }
        }
        ++it;
        s = it % C::NS; ph = (it / C::NS) & 1u; buf = it % C::NT;
      }
      if (!ok) break;
      // ---- write the tile: a lane's four pairs of a 32-column chunk are eight consecutive output columns ----
      const bool vec_ok = ((p.ldc & 7) == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0) && (ti.q0 + col_base + CW <= ti.q_lim);
      const bool pair_ok = ((p.ldc & 1) == 0) && ((reinterpret_cast<uintptr_t>(out) & 3) == 0);
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const int prow = ti.p0 + quad * 32 + 8 * a + lr;
        if (prow >= ti.p_lim) continue;
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          const float2* v = f + (a * NCH + c) * 4;
          const int q = ti.q0 + col_base + c * 32 + lq * 8;
          if (vec_ok) {
            *reinterpret_cast<uint4*>(out + (long long)prow * p.ldc + q) =
                make_uint4(pack_pair<__nv_bfloat16>(v[0]), pack_pair<__nv_bfloat16>(v[1]), pack_pair<__nv_bfloat16>(v[2]),
                           pack_pair<__nv_bfloat16>(v[3]));
          } else {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              store_pair<__nv_bfloat16, false>(out, p.ldc, prow, q + 2 * kk, ti.q_lim, v[kk], pair_ok);
          }
        }
      }
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before_sync();
  cluster_sync();   // neither CTA leaves while the other may still read its shared memory or arrive on its barriers
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc_cg2(tmem_base, 512);
  if (threadIdx.x == 0 && *abort_flag) atomicOr(p.status, 1u);
}

// ------------------------------------------------------------------------------------------
// Expansion of packed codes to e4m3
// ------------------------------------------------------------------------------------------
// Four nibbles (bits 0..15 of `sel`, sign bits cleared) -> e4m3 of 0..7 or, where `neg` has 0xFF bytes, of -8..-1.
__device__ __forceinline__ uint32_t codes_to_e4m3(uint32_t sel, uint32_t neg) {
  const uint32_t pos = __byte_perm(0x44403800u, 0x4E4C4A48u, sel);   // 0 1 2 3 | 4 5 6 7
  const uint32_t ng = __byte_perm(0xCACCCED0u, 0xB8C0C4C8u, sel);    // -8 -7 -6 -5 | -4 -3 -2 -1
  return (neg & ng) | (~neg & pos);
}
__device__ __forceinline__ void expand_word(uint32_t w, uint32_t& lo, uint32_t& hi) {
  const uint32_t m = w & 0x77777777u, w4 = w << 4;
  uint32_t nlo, nhi;   // sign bit of every nibble replicated over its byte (prmt with the sign mode)
  asm("prmt.b32 %0, %1, %2, 0xD9C8;" : "=r"(nlo) : "r"(w4), "r"(w));
  asm("prmt.b32 %0, %1, %2, 0xFBEA;" : "=r"(nhi) : "r"(w4), "r"(w));
  lo = codes_to_e4m3(m, nlo);
  hi = codes_to_e4m3(m >> 16, nhi);
}

// Chunk c (16 packed bytes) of a packed [G, rows, 64 B] operand -> 32 bytes of its e4m3 form [G, pitch, 128 B].
__device__ __forceinline__ void expand_chunk(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, long long c, int rows, int pitch,
                                             bool permute) {
  const long long slot = c >> 2;
  const int g = (int)(slot / pitch), r = (int)(slot - (long long)g * pitch), j = (int)c & 3;
  uint4 w = make_uint4(0, 0, 0, 0);
  if (r < rows) w = __ldg(reinterpret_cast<const uint4*>(src + ((long long)g * rows + r) * 64 + j * 16));
  uint4 x, y;
  expand_word(w.x, x.x, x.y); expand_word(w.y, x.z, x.w);
  expand_word(w.z, y.x, y.y); expand_word(w.w, y.z, y.w);
  uint4* at = reinterpret_cast<uint4*>(dst + ((long long)g * pitch + (permute ? qperm(r) : r)) * 128 + j * 32);
  at[0] = x;
  at[1] = y;
}

// Packed [G, rows, 64 B] of both operands -> e4m3 [G, pitch, 128 B], pitch = rows rounded up to 32 (Q rows of a 32-row
// block in the order qperm; the rows that fill up a block are zero).  A thread expands 16 packed bytes.
__global__ void __launch_bounds__(256) expand_e4m3_kernel(const uint8_t* a, const uint8_t* b,
                                                          int M, int m_pitch, int N, int n_pitch, int G, int weights_early,
                                                          uint8_t* __restrict__ ea, uint8_t* __restrict__ eb) {
  if (!weights_early) {   // behind a kernel that may have written the weights
    pdl_wait();
    pdl_fresh(b);
  }
  // the weights first: with weights_early they are there while the quantiser still works on the activations
  const long long ca = (long long)G * m_pitch * 4, cb = (long long)G * n_pitch * 4, step = (long long)gridDim.x * 256;
  long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  for (; i < cb; i += step) expand_chunk(b, eb, i, N, n_pitch, true);
  a = pdl_wait(a);
  pdl_trigger();
  for (; i < ca + cb; i += step) expand_chunk(a, ea, i - cb, M, m_pitch, false);
}

template <int BN, bool AZP>
static int launch_f8(const GemmParams& p, const CUtensorMap& tmP, const CUtensorMap& tmQ, int p_pitch, int q_pitch, int grid,
                     cudaStream_t st, PairLaunch* pl) {
  using C = F8Cfg<BN>;
  static_assert(C::SMEM_BYTES <= 232448, "shared memory layout exceeds the 227 KB a CTA may use");
  I4TC_CUDA(cudaFuncSetAttribute(w4a4_group_f8_kernel<BN, AZP>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid, 1, 1);
  cfg.blockDim = dim3(C::THREADS, 1, 1);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;   // (behind the expansion, whoever called)
  return launch_pairs(cfg, pl, w4a4_group_f8_kernel<BN, AZP>, p, tmP, tmQ, p_pitch, q_pitch);
}

long long group_f8_scratch_bytes(long long M, long long N, int G) {
  return (((M + 31) & ~31ll) + ((N + 31) & ~31ll)) * G * 128;
}

int launch_w4a4_group_f8(const GemmParams& p, const uint8_t* a, const uint8_t* b, uint8_t* scratch, int bn, int device,
                         int sm_count, cudaStream_t st, PairLaunch* pl) {
  const int M = p.P_rows, N = p.Q_rows;
  const int m_pitch = (M + 31) & ~31, n_pitch = (N + 31) & ~31;
  uint8_t* ea = scratch;
  uint8_t* eb = scratch + (long long)m_pitch * p.G * 128;
  CUtensorMap tmP, tmQ;
  if (int rc = get_tensor_map_i8(device, ea, (long long)m_pitch * p.G, 128, 128, &tmP)) return rc;
  if (int rc = get_tensor_map_i8(device, eb, (long long)n_pitch * p.G, 128, bn / 2, &tmQ)) return rc;
  const long long chunks = (long long)(m_pitch + n_pitch) * p.G * 4;
  const long long blocks = (chunks + 255) / 256, cap = (long long)sm_count * 8 * 4;
  I4TC_CUDA(launch_kernel(true, expand_e4m3_kernel, dim3((unsigned)(blocks < cap ? blocks : cap)), 256, 0, st, a, b, M, m_pitch,
                          N, n_pitch, p.G, p.weights_early, ea, eb));
  const long long tiles = (long long)p.num_p_tiles * p.num_q_tiles;
  const int grid = 2 * (int)(tiles < sm_count / 2 ? tiles : sm_count / 2);
  const bool azp = p.zp != nullptr;
  if (bn == 256) return azp ? launch_f8<256, true>(p, tmP, tmQ, m_pitch, n_pitch, grid, st, pl) : launch_f8<256, false>(p, tmP, tmQ, m_pitch, n_pitch, grid, st, pl);
  if (bn == 192) return azp ? launch_f8<192, true>(p, tmP, tmQ, m_pitch, n_pitch, grid, st, pl) : launch_f8<192, false>(p, tmP, tmQ, m_pitch, n_pitch, grid, st, pl);
  return azp ? launch_f8<128, true>(p, tmP, tmQ, m_pitch, n_pitch, grid, st, pl) : launch_f8<128, false>(p, tmP, tmQ, m_pitch, n_pitch, grid, st, pl);
}

}  // namespace i4tc

// Stacked-GEMM conv-attention backward on tcgen05 / TMEM / TMA for head dim 128 (entries off the
// causal band; the math is that of bwd_tc.cu).
//
// At d = 128 a stacked key tile is twice as large as at d = 64 and the accumulators twice as wide, so the
// plans of bwd_tc.cu do not fit the 227 KB of shared memory / 512 columns of tensor memory.  The kernel
// here keeps the query rows on the TMEM lanes for the scores (S = sum_a Q^(a) Kt_a^T, M = 128 rows, N = 64
// keys):
//
//   bwd_dkdv_tc128_kernel : CTA = 64 keys, loops 128-row query blocks.  The accumulators are kept TRANSPOSED, with the head
//                           dim on the lanes: dV^T[d, key] += dO^T P and dKt_a^T[d, key] += Q^(a)T dC are
//                           M = 128 MMAs whose A operand is the staged dO / Q tile read MN-major and whose B
//                           operand is the bf16 P / dC tile as the element-wise warps write it (one row per
//                           thread), dC with the tap's row shift as a start-address offset of 128 bytes per row
//                           into a 128-byte-swizzled tile: three taps are one MMA of 192 columns (blocks walked
//                           from the last one down; with the shift on Q, 64 columns each: 9.4 ms, now 7.9, at
//                           B 8, H 32, N 4096).  dV^T + 6 dKt^T take 448 columns; S and dP share the last 64
//                           (S(0) dP(0) | S(1) dP(1) | ...).  Scores and dP are computed once per entry.
//   Four of the stacked key tiles stay resident; the others and V come again for every block through a ring of three 8 KB
//   slabs, interleaved with the resident ones.  That is 48 KB per 128 x 64 block more from L2, and makes room for a second
//   Q tile, so that S of the next block runs under the dKt MMAs of this one: with everything resident and one Q tile the
//   block's load, S, element-wise part and dKt were one chain (tensor core 35 % busy, B 8, H 32, N 4096: 10.4 ms, then 9.4).
//   Bound by the shared-memory port: S (M = 128, N = 64) reads 6 KB for 32 cycles of arithmetic.
// Every mbarrier wait is bounded; no TMA multicast, no cluster, cta_group::1 only.
#include <cuda.h>
#include <cuda_runtime.h>

#include "bwd_tc.cuh"
#include "fmta_tc.cuh"
#include "launch_util.cuh"

namespace fmta {

// ==========================================================================================
// dK-tilde / dV, d = 128
// ==========================================================================================
struct Dkv128Cfg {
  static constexpr int D = 128;
  static constexpr int BK = 64;                // keys per CTA (= columns of the transposed accumulators)
  static constexpr int BR = 128;               // query rows per block (= TMEM lanes of S and dP)
  static constexpr int HALO = 8;               // pad_q <= 5
  static constexpr int QR = BR + HALO;         // rows of Q per block
  static constexpr int RES = 4;                // resident Kt tiles
  static constexpr int NST = 3;                // slabs of the ring for the other Kt tiles and V
  static constexpr int SLAB_BYTES = BK * 128;  // 64 keys x 64 elements, 128-byte swizzle
  static constexpr int KT_BYTES = 2 * SLAB_BYTES;
  static constexpr int DO_SLAB = BR * 128;     // 128 rows x 64 elements, 128-byte swizzle
  static constexpr int oKt = 0;
  static constexpr int oSt = oKt + RES * KT_BYTES;
  static constexpr int Q_SLAB = QR * 128;      // 136 rows x 64 elements, 128-byte swizzle
  static constexpr int oQ = oSt + NST * SLAB_BYTES;             // two buffers of two slabs
  static constexpr int odO = oQ + 4 * Q_SLAB;                   // two slabs
  static constexpr int oP = odO + 2 * DO_SLAB;                  // P  : [BK/8][BR][16 B]  (MN-major B operand)
  static constexpr int oDC = oP + (BK / 8) * BR * 16;           // dC : [136 rows][128 B], 128-byte swizzle
  static constexpr int oBar = oDC + QR * 128;
  static constexpr int kSmemBytes = oBar + 512 + 1024;
  static_assert(odO % 1024 == 0 && oDC % 1024 == 0 && oSt % 1024 == 0 && oQ % 1024 == 0 && Q_SLAB % 1024 == 0, "swizzled tiles start on 1024-byte boundaries");
  static_assert(kSmemBytes <= 227 * 1024, "dK/dV kernel (d = 128): shared memory budget");
  static constexpr int kTmemCols = 512;        // dV^T at 0, dKt_a^T at 64 (1 + a), scratch X (S / dP) at 448
  static constexpr int colX = 448;
  static constexpr int kEwWarps = 8;
  static constexpr int kThreads = (kEwWarps + 5) * 32;   // + issuer S, issuers A0 and A1, two producers
};

__global__ void __launch_bounds__(Dkv128Cfg::kThreads, 1)
bwd_dkdv_tc128_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
                      const __grid_constant__ CUtensorMap tmKt, const __grid_constant__ CUtensorMap tmV,
                      const BwdTcParams p) {
  using Cfg = Dkv128Cfg;
  constexpr int D = Cfg::D, BK = Cfg::BK, BR = Cfg::BR, HALO = Cfg::HALO, QR = Cfg::QR;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* sKt = smem + Cfg::oKt;
  unsigned char* sSt = smem + Cfg::oSt;
  unsigned char* sQ = smem + Cfg::oQ;
  unsigned char* sdO = smem + Cfg::odO;
  constexpr int NST = Cfg::NST;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::oBar);
  uint64_t* st_full = bars;              // [NST] slab of the ring staged
  uint64_t* st_empty = st_full + NST;    // [NST] slab read
  uint64_t* kt_full = st_empty + NST;    // resident Kt tiles staged
  uint64_t* q_full = kt_full + 1;        // [2] Q of the block staged
  uint64_t* q_free = q_full + 2;         // [2] the three issuers are done with it (3 commits)
  uint64_t* do_full = q_free + 2;        // dO of the block staged
  uint64_t* do_free = do_full + 1;       // dP and dV^T of the block have read it (2 commits)
  uint64_t* s_full = do_free + 1;        // S in X
  uint64_t* xs_free = s_full + 1;        // S taken into registers (256 arrivals): X free for dP
  uint64_t* dp_full = xs_free + 1;       // dP in X
  uint64_t* xd_free = dp_full + 1;       // dP taken into registers (256 arrivals): X free for the next S
  uint64_t* p_full = xd_free + 1;        // P (bf16) written to shared memory (256 arrivals)
  uint64_t* p_free = p_full + 1;         // the dV^T MMAs that read it have completed
  uint64_t* dc_full = p_free + 1;        // dC (bf16) written to shared memory (256 arrivals)
  uint64_t* dc_free = dc_full + 1;       // the dKt^T MMAs that read it have completed (2 commits)
  uint64_t* all_done = dc_free + 1;
  uint64_t* never_bar = all_done + 1;
  uint64_t* mma_drain = never_bar + 1;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(mma_drain + 1);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
  volatile int* s_q_issued = s_abort + 1;    // blocks whose Q / dO copies, slabs whose copies the producers have issued
  volatile int* s_do_issued = s_abort + 2;
  volatile int* s_st_issued = s_abort + 3;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int N = p.N, cq = p.cq, pq = cq - 1, pk = (p.ck - 1) / 2;
  const int band = pq + pk;
  int h, b, j0;
  dkdv_block_order(BK, h, b, j0);          // (batch, head)-major, key-tile-major tail
  j0 += p.key_base;
  const int bh = b * p.H + h;
  const int nQB = (N + BR - 1) / BR;
  // The blocks are walked from the last one down, as a block's dKt^T takes the first pad_q rows of dC of the block behind it.
  // No block in front of the last one walked misses its own: the first pad_q rows there are not owned (j0 + band is the first
  // owned row), or there is nothing in front of it.
  const int qb_begin = p.causal ? min(nQB, (j0 + pk) / BR) : 0;
  const int nblk = nQB - qb_begin;

  if (tid == 0) {
    for (int i = 0; i < NST; ++i) { tc::mbar_init(&st_full[i], 1); tc::mbar_init(&st_empty[i], 1); }
    tc::mbar_init(kt_full, 1);
    for (int i = 0; i < 2; ++i) { tc::mbar_init(&q_full[i], 1); tc::mbar_init(&q_free[i], 3); }
    tc::mbar_init(do_full, 1); tc::mbar_init(do_free, 2);
    tc::mbar_init(s_full, 1); tc::mbar_init(xs_free, Cfg::kEwWarps * 32);
    tc::mbar_init(dp_full, 1); tc::mbar_init(xd_free, Cfg::kEwWarps * 32);
    tc::mbar_init(p_full, Cfg::kEwWarps * 32); tc::mbar_init(p_free, 1);
    tc::mbar_init(dc_full, Cfg::kEwWarps * 32); tc::mbar_init(dc_free, 2);
    tc::mbar_init(all_done, 2);
    tc::mbar_init(never_bar, 1); tc::mbar_init(mma_drain, 3);
    *s_abort = 0; *s_q_issued = 0; *s_do_issued = 0; *s_st_issued = 0;
    tc::mbar_fence_init();
  }
  if (warp == Cfg::kEwWarps) {
    tc::tmem_alloc(s_tmem, Cfg::kTmemCols);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  pdl_trigger();
  __syncthreads();   // no pdl_wait() here: see the d = 64 kernel
  tc::tc_fence_after();
  const uint32_t tmem = *s_tmem;
  const uint32_t tX = tmem + Cfg::colX;

  const int role = warp - Cfg::kEwWarps;       // 0: issuer S, 1, 2: issuers A0, A1, 3: producer of Kt, Q and dO, 4: of the ring
  const int nres = min(cq, Cfg::RES);

  if (role == 3) {
    if (nblk > 0 && lane == 0) {
      tc::tma_prefetch_desc(&tmQ); tc::tma_prefetch_desc(&tmdO); tc::tma_prefetch_desc(&tmKt);
      auto load_q = [&](int it) {
        uint64_t* bar = &q_full[it & 1];
        unsigned char* dst = sQ + (it & 1) * (2 * Cfg::Q_SLAB);
        const int i0 = (nQB - 1 - it) * BR;
        tc::mbar_expect_tx(bar, QR * D * 2);
        tc::tma_load_3d(dst, &tmQ, bar, 0, i0 - HALO, bh);
        tc::tma_load_3d(dst + Cfg::Q_SLAB, &tmQ, bar, 64, i0 - HALO, bh);
        *s_q_issued = it + 1;
      };
      load_q(0);
      tc::mbar_expect_tx(kt_full, nres * Cfg::KT_BYTES);
      for (int a = 0; a < nres; ++a) {
        tc::tma_load_3d(sKt + a * Cfg::KT_BYTES, &tmKt, kt_full, 0, j0, bh * cq + a);
        tc::tma_load_3d(sKt + a * Cfg::KT_BYTES + Cfg::SLAB_BYTES, &tmKt, kt_full, 64, j0, bh * cq + a);
      }
      for (int it = 0; it < nblk; ++it) {
        const int i0 = (nQB - 1 - it) * BR;
        if (it > 0 && !tc::mbar_wait(do_free, (it - 1) & 1, s_abort)) break;                     // dP and dV of block it-1
        tc::mbar_expect_tx(do_full, 2 * Cfg::DO_SLAB);
        tc::tma_load_3d(sdO, &tmdO, do_full, 0, i0, bh);
        tc::tma_load_3d(sdO + Cfg::DO_SLAB, &tmdO, do_full, 64, i0, bh);
        *s_do_issued = it + 1;
        if (it + 1 < nblk) {
          if (it > 0 && !tc::mbar_wait(&q_free[(it + 1) & 1], ((it - 1) >> 1) & 1, s_abort)) break;   // everything of block it-1
          load_q(it + 1);
        }
      }
    }
  } else if (role == 4) {
    // the ring, in the order of the issuer: the slabs of the taps that are not resident, then V
    if (nblk > 0 && lane == 0) {
      tc::tma_prefetch_desc(&tmV);
      const int per = 2 * (cq - nres) + 2;
      int slot = 0, ph = 1, id = 0;
      bool ok = true;
      for (int it = 0; it < nblk && ok; ++it)
        for (int i = 0; i < per; ++i) {
          if (!(ok = tc::mbar_wait(&st_empty[slot], ph, s_abort))) break;
          tc::mbar_expect_tx(&st_full[slot], Cfg::SLAB_BYTES);
          const bool is_v = i >= per - 2;
          tc::tma_load_3d(sSt + slot * Cfg::SLAB_BYTES, is_v ? &tmV : &tmKt, &st_full[slot], (i & 1) * 64, j0, is_v ? bh : bh * cq + nres + (i >> 1));
          if (++slot == NST) { slot = 0; ph ^= 1; }
          *s_st_issued = ++id;
        }
    }
  } else if (role == 0) {
    // ===================== MMA issuer S: S and dP of block `it` into the scratch columns X =====================
    if (nblk > 0) {   // all lanes run the loop; one elected lane issues
      constexpr uint32_t idescT = tc::make_idesc(BR, BK, 0, 0);    // 128 x 64, K-major operands
      const uint64_t dKtB = tc::make_sdesc(smem_u32(sKt), 16, 1024, tc::kLayoutSW128);
      const uint32_t hi = (uint32_t)(dKtB >> 32), kt_lo = (uint32_t)dKtB;
      const uint32_t ring_lo = kt_lo + (uint32_t)((Cfg::oSt - Cfg::oKt) >> 4), o_lo = kt_lo + (uint32_t)((Cfg::odO - Cfg::oKt) >> 4);
      // Q^(a), K-major: the same swizzled tile with the start address moved down by the tap's row shift.  The
      // tensor core applies the 128-byte swizzle to the absolute shared-memory address, exactly as TMA did when
      // it wrote the tile, so a start that is a multiple of 128 bytes (not of the 1024-byte pattern) reads the
      // shifted rows correctly.
      const uint32_t q_lo0 = kt_lo + (uint32_t)((Cfg::oQ - Cfg::oKt + (HALO - pq) * 128) >> 4);
      int slot = 0, ph = 0;
      bool ok = tc::mbar_wait_warp(kt_full, 0, s_abort);
      bool ready = false;                                          // the ring's next slab was seen staged (a wait that is
                                                                   // over already costs 200 cycles)
      auto slab = [&](uint32_t a_lo, uint32_t acc) {               // 64 contraction columns against the ring's next slab
        if (!ready && !(ok = tc::mbar_wait_warp(&st_full[slot], ph, s_abort))) return;
        tc::tc_fence_after();
        const int ns = slot + 1 == NST ? 0 : slot + 1, nph = ns == 0 ? ph ^ 1 : ph;
        const uint32_t seen = tc::mbar_test(&st_full[ns], nph);
        tc::mma4_ss(tX, a_lo, hi, 2, ring_lo + (uint32_t)(slot * (Cfg::SLAB_BYTES >> 4)), hi, 2, idescT, acc);
        tc::mma_commit_e(&st_empty[slot]);
        slot = ns; ph = nph;
        ready = __all_sync(0xffffffffu, seen);
      };
      for (int it = 0; it < nblk && ok; ++it) {
        ok = tc::mbar_wait_warp(&q_full[it & 1], (it >> 1) & 1, s_abort);
        if (ok && it > 0) ok = tc::mbar_wait_warp(xd_free, (it - 1) & 1, s_abort);       // dP(it-1) has left X
        if (!ok) break;
        tc::tc_fence_after();
        // S = sum_a Q^(a) Kt_a^T: one slab of the ring, two resident ones, ...
        const uint32_t q_lo = q_lo0 + (uint32_t)((it & 1) * (2 * Cfg::Q_SLAB >> 4));
        const int ns = 2 * (cq - nres), nr = 2 * nres;
        for (int i = 0; i < max(ns, nres) && ok; ++i) {
          if (i < ns) slab(q_lo + (uint32_t)((i & 1) * (Cfg::Q_SLAB >> 4) + (nres + (i >> 1)) * (128 >> 4)), i != 0);
          if (!ok) break;
          if (2 * i < nr) {
#pragma unroll
            for (int sl = 0; sl < 2; ++sl)
              tc::mma4_ss(tX, q_lo + (uint32_t)(sl * (Cfg::Q_SLAB >> 4) + i * (128 >> 4)), hi, 2,
                          kt_lo + (uint32_t)((i * Cfg::KT_BYTES + sl * Cfg::SLAB_BYTES) >> 4), hi, 2, idescT, ns > 0 || i + sl != 0);
          }
        }
        if (!ok) break;
        tc::mma_commit_e(s_full);
        tc::mma_commit_e(&q_free[it & 1]);
        ok = tc::mbar_wait_warp(do_full, it & 1, s_abort);
        if (ok) ok = tc::mbar_wait_warp(xs_free, it & 1, s_abort);                       // S(it) has left X
        if (!ok) break;
        tc::tc_fence_after();
        slab(o_lo, 0);                                                                   // dP = dO V^T
        if (ok) slab(o_lo + (uint32_t)(Cfg::DO_SLAB >> 4), 1);
        if (!ok) break;
        tc::mma_commit_e(dp_full);
        tc::mma_commit_e(do_free);
      }
    }
  } else if (role > 0) {
    // ===================== MMA issuers A0 / A1: dV^T += dO^T P ; dKt_a^T += Q^T dC^(a) =====================
    // The tap's row shift is on dC, whose rows are the contraction: dKt_a[j] = sum_i q_i dC[i + s, j], s = pad_q - a.  Three taps
    // then share their A operand: three 64-key atoms of B that start one row (128 bytes) apart are one MMA of 192 columns.
    // With the shift on Q each tap was an MMA of its own, whose 4 KB of Q take as long to read as 64 columns to multiply.
    const int ai = role - 1;
    if (nblk > 0) {   // all lanes run the loop; one elected lane issues
      constexpr uint32_t idescA = tc::make_idesc(D, BK, 1, 1);     // 128 (head dim) x 64 (keys), both operands MN-major
      // A0 takes dV^T and the first half of the shifts, A1 the rest (c_q <= 6: at most three)
      const int accb = p.with_dv ? 1 : 0;
      const int s_begin = ai == 0 ? 0 : cq / 2, ns = ai == 0 ? cq / 2 : cq - cq / 2;
      const uint32_t idescK = tc::make_idesc(D, BK * ns, 1, 1);
      // dO read MN-major (M = head dim across the two slabs, K = rows): 16 rows = 2048 bytes per step
      const uint64_t dOm = tc::make_sdesc(smem_u32(sdO), Cfg::DO_SLAB, 1024, tc::kLayoutSW128);
      // Q read MN-major (M = head dim across the two slabs, K = rows)
      const uint64_t dQm = tc::make_sdesc(smem_u32(sQ) + HALO * 128, Cfg::Q_SLAB, 1024, tc::kLayoutSW128);
      // dC: N = 64 keys per shift, one row apart, K = rows
      const uint64_t dCb = tc::make_sdesc(smem_u32(smem + Cfg::oDC) + s_begin * 128, 128, 1024, tc::kLayoutSW128);
      // P: N = keys in 8-key chunks BR * 16 bytes apart, K = rows 16 bytes apart
      const uint64_t dPb = tc::make_sdesc(smem_u32(smem + Cfg::oP), 128, BR * 16, tc::kLayoutNone);
      const uint32_t om_hi = (uint32_t)(dOm >> 32), om_lo = (uint32_t)dOm;
      const uint32_t qm_hi = (uint32_t)(dQm >> 32), qm_lo0 = (uint32_t)dQm;
      const uint32_t pb_hi = (uint32_t)(dPb >> 32), pb_lo = (uint32_t)dPb, cb_hi = (uint32_t)(dCb >> 32), cb_lo = (uint32_t)dCb;
      bool ok = true;
      for (int it = 0; it < nblk && ok; ++it) {
        const uint32_t acc_on = it != 0;
        if (ai == 0) {
          ok = tc::mbar_wait_warp(do_full, it & 1, s_abort) && tc::mbar_wait_warp(p_full, it & 1, s_abort);
          if (!ok) break;
          tc::tc_fence_after();
          if (p.with_dv) {
            tc::mma4_ss(tmem, om_lo, om_hi, 2048 / 16, pb_lo, pb_hi, 16, idescA, acc_on);
            tc::mma4_ss(tmem, om_lo + 4 * (2048 / 16), om_hi, 2048 / 16, pb_lo + 4 * 16, pb_hi, 16, idescA, 1);
          }
          tc::mma_commit_e(do_free);
          tc::mma_commit_e(p_free);
        }
        ok = tc::mbar_wait_warp(&q_full[it & 1], (it >> 1) & 1, s_abort) && tc::mbar_wait_warp(dc_full, it & 1, s_abort);
        if (!ok) break;
        tc::tc_fence_after();
        const uint32_t qm_lo = qm_lo0 + (uint32_t)((it & 1) * (2 * Cfg::Q_SLAB >> 4));
        // A1's taps go behind S of the next block, which would otherwise share the tensor core with all of them from its
        // first MMA on and end with nothing left to run while it is taken out of X
        if (ai == 1 && it + 1 < nblk && !tc::mbar_wait_warp(s_full, (it + 1) & 1, s_abort)) { ok = false; break; }
        if (ns > 0) {
          const uint32_t dst = tmem + 64 * (accb + s_begin);
          tc::mma4_ss(dst, qm_lo, qm_hi, 2048 / 16, cb_lo, cb_hi, 2048 / 16, idescK, acc_on);
          tc::mma4_ss(dst, qm_lo + 4 * (2048 / 16), qm_hi, 2048 / 16, cb_lo + 4 * (2048 / 16), cb_hi, 2048 / 16, idescK, 1);
        }
        tc::mma_commit_e(&q_free[it & 1]);
        tc::mma_commit_e(dc_free);
      }
      if (ok) tc::mma_commit_e(all_done);
    }
  } else {
    // ===================== element-wise warps: query row = lane, CW keys per thread =====================
    constexpr int NCG = Cfg::kEwWarps / 4, CW = BK / NCG;     // column groups (warps per lane quarter), columns each
    const int qtr = warp & 3, cg = warp >> 2;
    const int row = qtr * 32 + lane;
    const uint32_t lane_base = (uint32_t)(qtr * 32) << 16;
    const uint32_t tXl = tX + lane_base + CW * cg;
    bool ok = true;
    // every thread fetches the statistics of its own row (LSE in log2 units, D), one block ahead
    float lse2 = 0.f, dvec = 0.f;
    uint32_t above[CW / 2];                             // dC of this row of the block before, which lies behind this one
#pragma unroll
    for (int c = 0; c < CW / 2; ++c) above[c] = 0u;
    if (nblk > 0) {
      const int gi = (nQB - 1) * BR + row;
      if (gi < N) { lse2 = p.LSE[(size_t)bh * N + gi] * kLog2e; dvec = p.Dvec[(size_t)bh * N + gi]; }
    }
    for (int it = 0; it < nblk && ok; ++it) {
      const int i0 = (nQB - 1 - it) * BR;
      const int gi = i0 + row;
      float lse2_next = 0.f, dvec_next = 0.f;
      if (it + 1 < nblk) {                              // (every row of a block but the last is a row of the sequence)
        lse2_next = p.LSE[(size_t)bh * N + gi - BR] * kLog2e;
        dvec_next = p.Dvec[(size_t)bh * N + gi - BR];
      }
      ok = __all_sync(0xffffffffu, (p.selftest_expire && it == 0) ? tc::mbar_wait(never_bar, 0, s_abort, tc::kSelfTestSpinLimit)
                                                                  : tc::mbar_wait(s_full, it & 1, s_abort));
      if (!ok) break;
      tc::tc_fence_after();
      float s[CW];
      tc::tmem_ldn(tXl, s);
      tc::tc_fence_before();
      tc::mbar_arrive(xs_free);
      // P[i, key] = exp2(S - LSE_i), kept only where this kernel owns the entry; dC = P (dP - D_i)
      uint32_t pp[CW / 2];
      const int kbase = j0 + CW * cg;
      if ((j0 + BK <= N) && (i0 + BR <= N) && (!p.causal || j0 + BK - 1 + band <= i0)) {   // block owned entirely
#pragma unroll
        for (int c = 0; c < CW; ++c) s[c] = exp2f(s[c] - lse2);
      } else {
        const int jlim = (gi < N) ? (p.causal ? min(N - 1, gi - band) : N - 1) : -1;   // last key this row owns here
#pragma unroll
        for (int c = 0; c < CW; ++c) s[c] = (kbase + c <= jlim) ? exp2f(s[c] - lse2) : 0.f;
      }
#pragma unroll
      for (int c = 0; c < CW; c += 2) pp[c / 2] = pack_bf16(s[c], s[c + 1]);
      if (it > 0) {   // dV^T of block it-1 has finished reading P
        ok = __all_sync(0xffffffffu, tc::mbar_wait(p_free, (it - 1) & 1, s_abort));
        if (!ok) break;
      }
      unsigned char* pt = smem + Cfg::oP + row * 16;
      unsigned char* dc = smem + Cfg::oDC + row * 128;
#pragma unroll
      for (int q4 = 0; q4 < CW / 8; ++q4)            // 8 keys (16 bytes) per chunk
        *reinterpret_cast<uint4*>(pt + ((CW / 8) * cg + q4) * (BR * 16)) = make_uint4(pp[4 * q4], pp[4 * q4 + 1], pp[4 * q4 + 2], pp[4 * q4 + 3]);
      tc::fence_proxy_async_smem();
      tc::mbar_arrive(p_full);
      ok = __all_sync(0xffffffffu, tc::mbar_wait(dp_full, it & 1, s_abort));
      if (!ok) break;
      tc::tc_fence_after();
      float dp[CW];
      tc::tmem_ldn(tXl, dp);
      tc::tc_fence_before();
      tc::mbar_arrive(xd_free);
#pragma unroll
      for (int c = 0; c < CW; c += 2) pp[c / 2] = pack_bf16(s[c] * (dp[c] - dvec), s[c + 1] * (dp[c + 1] - dvec));
      if (it > 0) {   // dKt^T of block it-1 has finished reading dC
        ok = __all_sync(0xffffffffu, tc::mbar_wait(dc_free, (it - 1) & 1, s_abort));
        if (!ok) break;
      }
#pragma unroll
      for (int q4 = 0; q4 < CW / 8; ++q4)
        *reinterpret_cast<uint4*>(dc + ((((CW / 8) * cg + q4) ^ (row & 7)) << 4)) = make_uint4(pp[4 * q4], pp[4 * q4 + 1], pp[4 * q4 + 2], pp[4 * q4 + 3]);
      if (row < HALO) {
#pragma unroll
        for (int q4 = 0; q4 < CW / 8; ++q4)
          *reinterpret_cast<uint4*>(dc + BR * 128 + ((((CW / 8) * cg + q4) ^ (row & 7)) << 4)) =
              make_uint4(above[4 * q4], above[4 * q4 + 1], above[4 * q4 + 2], above[4 * q4 + 3]);
      }
#pragma unroll
      for (int c = 0; c < CW / 2; ++c) above[c] = pp[c];
      tc::fence_proxy_async_smem();
      tc::mbar_arrive(dc_full);
      lse2 = lse2_next; dvec = dvec_next;
    }
    // ---- epilogue: the accumulators hold dV^T and dKt_a^T (lane = head dim, column = key); chunks of 32
    // keys are dealt round-robin to the two column groups ----
    if (nblk > 0 && ok) ok = __all_sync(0xffffffffu, tc::mbar_wait(all_done, 0, s_abort));
    tc::tc_fence_after();
    const bool have = (nblk > 0) && ok;
    const int nacc = (p.with_dv ? 1 : 0) + p.ntap;
    pdl_wait();                                         // the band kernel's part of dV
    const int dcol = qtr * 32 + lane;                   // head-dim index of this lane
    for (int ch = cg; ch < 2 * nacc; ch += NCG) {
      const int acc = ch >> 1, half = ch & 1;
      float o[32];
      if (have) {
        tc::tmem_ld32(tmem + lane_base + ch * 32, o);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = 0.f;
      }
      const int key0 = j0 + half * 32;
      if (p.with_dv && acc == 0) {
        const size_t at = ((size_t)bh * N + key0) * D + dcol;        // a warp touches 32 consecutive elements per key
        if (p.dVadd) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (key0 + i < N) o[i] += p.dVadd[at + (size_t)i * D];
        }
        if (p.out_bf16) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (key0 + i < N) reinterpret_cast<bf16*>(p.dV)[at + (size_t)i * D] = __float2bfloat16(o[i]);
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (key0 + i < N) reinterpret_cast<float*>(p.dV)[at + (size_t)i * D] = o[i];
        }
      } else {
        // dKt_a leaves as bf16 [key][d]: neighbouring lanes pair up so that every lane stores one 4-byte word
        const int tap = cq - 1 - (acc - (p.with_dv ? 1 : 0));      // accumulators in the order of the shifts
        bf16* dst = p.dKt + (((size_t)bh * cq + tap) * N + key0) * D + (dcol & ~1);
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float mine_even = o[i], mine_odd = o[i + 1];
          const float other_even = __shfl_xor_sync(0xffffffffu, mine_even, 1);
          const float other_odd = __shfl_xor_sync(0xffffffffu, mine_odd, 1);
          // even lane: key i, columns (dcol, dcol + 1); odd lane: key i + 1, columns (dcol - 1, dcol)
          const bool odd = lane & 1;
          const uint32_t w = odd ? pack_bf16(other_odd, mine_odd) : pack_bf16(mine_even, other_even);
          const int key = key0 + i + (odd ? 1 : 0);
          if (key < N) *reinterpret_cast<uint32_t*>(dst + (size_t)(i + (odd ? 1 : 0)) * D) = w;
        }
      }
    }
  }
  __syncwarp();

  tc::tc_fence_before();
  __syncthreads();
  if (*s_abort) {
    if (tid == 0) atomicExch(p.status, 1);
    // MMAs and copies of this CTA are waited for (bounded) before its memories go
    if (role >= 0 && role < 3) tc::mma_commit_e(mma_drain);
    if (role == 3 && lane == 0) {
      volatile int never = 0;
      if (nblk > 0) {
        const int qi = *s_q_issued, di = *s_do_issued, si = *s_st_issued;
        tc::mbar_wait(kt_full, 0, &never);
        for (int it = max(0, qi - 2); it < qi; ++it) tc::mbar_wait(&q_full[it & 1], (it >> 1) & 1, &never);
        if (di > 0) tc::mbar_wait(do_full, (di - 1) & 1, &never);
        for (int id = max(0, si - NST); id < si; ++id) tc::mbar_wait(&st_full[id % NST], (id / NST) & 1, &never);
      }
      tc::mbar_wait(mma_drain, 0, &never);
    }
    __syncthreads();
  }
  if (warp == Cfg::kEwWarps) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, Cfg::kTmemCols);
  }
}

// ==========================================================================================
// host side
// ==========================================================================================
cudaError_t launch_bwd_dkdv_tc128(const TrainParams& p, const __nv_bfloat16* Kt, __nv_bfloat16* dKt, int* status, int with_dv,
                                  int key_lo, int key_hi, cudaStream_t stream) {
  using Cfg = Dkv128Cfg;
  constexpr int D = Cfg::D;
  const size_t BH = (size_t)p.B * p.H;
  alignas(64) CUtensorMap tmQ, tmdO, tmKt, tmV;
  if (!make_tensor_map_bf16(&tmQ, p.Q, D, p.N, BH, 64, Cfg::QR, true)) return cudaErrorInvalidValue;
  if (!make_tensor_map_bf16(&tmdO, p.dO, D, p.N, BH, 64, Cfg::BR, true)) return cudaErrorInvalidValue;
  if (!make_tensor_map_bf16(&tmKt, Kt, D, p.N, BH * p.cq, 64, Cfg::BK, true)) return cudaErrorInvalidValue;
  if (!make_tensor_map_bf16(&tmV, p.V, D, p.N, BH, 64, Cfg::BK, true)) return cudaErrorInvalidValue;
  BwdTcParams bp = {};
  bp.LSE = p.LSE; bp.Dvec = p.Dvec; bp.dV = p.dVo; bp.dVadd = p.causal ? p.dV : nullptr; bp.out_bf16 = p.grad_bf16; bp.dKt = dKt; bp.status = status;
  bp.B = p.B; bp.H = p.H; bp.N = p.N; bp.cq = p.cq; bp.ck = p.ck; bp.causal = p.causal;
  bp.ntap = p.cq; bp.with_dv = with_dv;
  bp.key_base = key_lo;
  bp.selftest_expire = take_selftest_expire(kKernBwdDkdvTc);
  auto kern = bwd_dkdv_tc128_kernel;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
  if (e != cudaSuccess) return e;
  dim3 grid((key_hi - key_lo + Cfg::BK - 1) / Cfg::BK, p.H, p.B);
  return launch_pdl(kern, grid, dim3(Cfg::kThreads), Cfg::kSmemBytes, stream, tmQ, tmdO, tmKt, tmV, bp);
}

}  // namespace fmta

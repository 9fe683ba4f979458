// dQ of the stacked-GEMM backward on CTA pairs (the math of bwd_tc.cu; entries off the causal band):
//     C = sum_a Q^(a) Kt_a^T,  P = exp2(C - LSE*log2e),  dC = P * (dO V^T - D),  dQ[i'] = ln2 * sum_a sum_j dC[i' + pad_q - a, j] Kt_a[j]
//
// A pair of CTAs walks blocks of 128 keys for 256 rows of dC (a tile of 128 per CTA, one TMEM lane per row).  A
// tile computes 128 dC rows but owns only the first 128 - pad_q as dQ rows: dQ row i' needs dC rows i'..i'+pad_q, so tiles
// overlap by pad_q rows (recomputed) and no dQ row is shared.  The row shifts of Q and dC are free: both are staged as
// 128-byte-swizzled tiles and the tensor core applies the swizzle to the absolute shared-memory address, so a view shifted
// by s rows starts 128 s bytes further.
//   S, dP : 256 x 128 x 16 MMAs, each CTA stages half the KEYS of every Kt and V tile;
//   dQ    : 256 x d x 16 MMAs, each CTA stages half the COLUMNS of every Kt tile (a second copy, fetched just in time
//           instead of being held from S to dQ).
// Scores (S, dP) and dQ are two streams with an issuing warp, a TMA warp and a ring of tiles each: the tensor core takes an
// MMA only when the one before it is under way, so what one issuer does between two tiles (190 cycles) leaves it idle unless
// the other has MMAs waiting.
// Measured (B200, c_q 6, causal, N 4096; single CTAs before): d = 128, B 8, H 32: 7.8 -> 5.1 ms; d = 64, B 4, H 16: 831 ->
// 800 us; d = 64, N 1024, 8 heads, c_q 7: 63 -> 33 us.  Two row tiles per CTA (d = 64, S and dP taking turns in one set of
// columns) move half the key tiles but took 864 us.  Bound by shared-memory operand reads: 5 KB per 43-cycle dQ MMA at d = 64.
// Every mbarrier wait is bounded; on expiry the status word is set and the pair drains and leaves.  No TMA multicast.
#include <cuda.h>
#include <cuda_runtime.h>

#include "bwd_tc.cuh"
#include "fmta_tc.cuh"
#include "launch_util.cuh"

namespace fmta {

template <int D>
struct DqCfg {
  static constexpr int BM = 128, BC = 128;
  static constexpr int HALO = 8;                                // rows of Q staged above a tile (pad_q <= 8)
  static constexpr int SLABS = D / 64;                          // 64-element (128-byte) column slabs per row
  static constexpr int Q_SLAB = (BM + HALO) * 128, Q_TILE = SLABS * Q_SLAB;
  static constexpr int O_SLAB = BM * 128, O_TILE = SLABS * O_SLAB;
  // dC: 64-key slabs of [136 rows][128 B]; the 8 rows below the tile are read by the shifted views of rows that are not owned
  static constexpr int C_SLAB = (BM + 8) * 128, C_TILE = 2 * C_SLAB;
  // ring tile: SLABS x [64 keys][64 elements] of Kt or V for S / dP; [128 keys][32] (d = 64) or 2 x [64 keys][64] (d = 128)
  // of Kt for dQ
  static constexpr int TILE_BYTES = D * 128;
  static constexpr int oQ = 0, oO = oQ + Q_TILE, oC = oO + O_TILE, oRing = oC + C_TILE;
  static_assert(Q_SLAB % 1024 == 0 && C_SLAB % 1024 == 0, "swizzled tiles start on 1024-byte boundaries");
  static constexpr int NSLOT = (227 * 1024 - 1024 - 512 - oRing) / TILE_BYTES, NSS = (NSLOT + 1) / 2, NSD = NSLOT - NSS;
  static constexpr int oBar = oRing + NSLOT * TILE_BYTES;
  static constexpr int kSmemBytes = oBar + 512 + 1024;
  static constexpr int colS = 0, colP = 128, colQ = 256;
  static constexpr int kTmemCols = 512;
  static constexpr int kEw = 8;                                 // element-wise warps: 4 lane quarters x 2 key halves
  static constexpr int kThreads = (kEw + 4) * 32;               // + TMA and MMA warp of the scores, of dQ
  static_assert(NSD >= 3 && kSmemBytes <= 227 * 1024, "shared memory budget");
  static_assert((2 * NSLOT + 9) * 8 + 16 <= 512, "barriers");
};

template <int D>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(DqCfg<D>::kThreads, 1)
bwd_dq_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO, const __grid_constant__ CUtensorMap tmKt,
                 const __grid_constant__ CUtensorMap tmKd, const __grid_constant__ CUtensorMap tmV, const BwdTcParams p) {
  using Cfg = DqCfg<D>;
  constexpr int BM = Cfg::BM, BC = Cfg::BC, HALO = Cfg::HALO, SLABS = Cfg::SLABS, NSLOT = Cfg::NSLOT, NSS = Cfg::NSS, EW = Cfg::kEw;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* sRing = smem + Cfg::oRing;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::oBar);
  // (rank 0): only the copy in rank 0's shared memory is used
  uint64_t* full = bars;                 // [NSLOT]  TMA of both CTAs -> MMA (rank 0); the first NSS are the scores' ring
  uint64_t* empty = bars + NSLOT;        // [NSLOT]  MMA -> TMA
  uint64_t* q_full = bars + 2 * NSLOT;   // Q and dO staged (rank 0)
  uint64_t* s_full = q_full + 1;         // S ready
  uint64_t* s_free = s_full + 1;        // S taken into registers (rank 0)
  uint64_t* p_full = s_free + 1;        // dP ready
  uint64_t* p_free = p_full + 1;        // dP taken into registers (rank 0)
  uint64_t* dc_full = p_free + 1;       // dC written to shared memory (rank 0)
  uint64_t* dq_done = dc_full + 1;      // dQ MMAs of the block complete (dC buffer reusable)
  uint64_t* never_bar = dq_done + 1;    // nothing arrives here (expiry self-test)
  uint64_t* mma_drain = never_bar + 1;   // abort path: the issued MMAs have completed (both issuers)
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(mma_drain + 1);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
  volatile int* s_issued = s_abort + 1;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = tc::cluster_rank();
  const int N = p.N, cq = p.cq, pq = cq - 1, pk = (p.ck - 1) / 2;
  const int band = pq + pk;
  const int OWN = p.own, rows_per_pair = OWN * 2;
  const int nQB = (p.row_end - p.row_base + rows_per_pair - 1) / rows_per_pair;
  int bh, qb;
  tc::pair_block_order(blockIdx.x >> 1, nQB, p.B * p.H, bh, qb);
  // Row blocks are laid out from the END of the rows: when their number is not a multiple of the block, the partly filled
  // block is the first one, which sees the fewest keys.  Its rows before row_base are computed (negative rows as zero
  // rows) and not stored.  CTA r's tile starts at row R0 + r OWN.
  const int R0 = p.row_end - (qb + 1) * rows_per_pair;
  const int nKB = (N + BC - 1) / BC;
  int nkb = nKB;
  if (p.causal) {                                        // key blocks with at least one key j <= (last row) - band
    const int last = min(N - 1, R0 + OWN + BM - 1) - band;
    nkb = last >= 0 ? min(nKB, last / BC + 1) : 0;
  }

  if (tid == 0) {
    for (int i = 0; i < NSLOT; ++i) { tc::mbar_init(&full[i], 1); tc::mbar_init(&empty[i], 1); }
    tc::mbar_init(q_full, 1);
    tc::mbar_init(s_full, 1); tc::mbar_init(s_free, 2 * EW);
    tc::mbar_init(p_full, 1); tc::mbar_init(p_free, 2 * EW);
    tc::mbar_init(dc_full, 2 * EW); tc::mbar_init(dq_done, 1);
    tc::mbar_init(never_bar, 1); tc::mbar_init(mma_drain, 2);
    *s_abort = 0; s_issued[0] = 0; s_issued[1] = 0;
    tc::mbar_fence_init();
  }
  if (warp == EW + 1) tc::tmem_alloc_pair(s_tmem, Cfg::kTmemCols);
  tc::tc_fence_before();
  tc::cluster_sync_all();
  // Behind the band kernel (p.early) everything but its part of dQ is complete already: the kernel starts under the
  // band kernel's tail and waits in its epilogue.  Otherwise it waits here.  The dK/dV kernel behind it starts as soon as
  // every CTA here has triggered and reads what was complete by then (all but this kernel's dQ), hence the order.
  if (!p.early) pdl_wait();
  pdl_trigger();
  tc::tc_fence_after();
  const uint32_t tmem = *s_tmem;
  const int role = warp - EW;                // 0, 1: TMA and MMA of the scores, 2, 3: of dQ

  if (role == 0 || role == 2) {
    // ===================== TMA producers: this CTA's Q and dO, its half of every Kt and V tile =====================
    if (lane == 0 && nkb > 0) {
      const bool is_s = role == 0;
      const int base = is_s ? 0 : NSS, n = is_s ? NSS : NSLOT - NSS;
      const uint32_t full0 = tc::cluster_addr(full, 0);
      if (is_s) {
        tc::tma_prefetch_desc(&tmQ); tc::tma_prefetch_desc(&tmdO); tc::tma_prefetch_desc(&tmKt); tc::tma_prefetch_desc(&tmV);
        const uint32_t qf = tc::cluster_addr(q_full, 0);
        if (rank == 0) tc::mbar_expect_tx(q_full, 2 * (Cfg::Q_TILE + Cfg::O_TILE));
        for (int sl = 0; sl < SLABS; ++sl) {
          tc::tma_load_3d_pair(smem + Cfg::oQ + sl * Cfg::Q_SLAB, &tmQ, qf, sl * 64, R0 + (int)rank * OWN - HALO, bh);
          tc::tma_load_3d_pair(smem + Cfg::oO + sl * Cfg::O_SLAB, &tmdO, qf, sl * 64, R0 + (int)rank * OWN, bh);
        }
      } else tc::tma_prefetch_desc(&tmKd);
      int slot = base, ph = 1, id = 0;
      bool ok = true;
      auto put = [&](const CUtensorMap* map, int x0, int dx, int y0, int dy, int z) {      // SLABS boxes of 8 KB
        if (!tc::mbar_wait(&empty[slot], ph, s_abort)) { ok = false; return; }
        if (rank == 0) tc::mbar_expect_tx(&full[slot], 2 * Cfg::TILE_BYTES);
#pragma unroll
        for (int i = 0; i < SLABS; ++i)
          tc::tma_load_3d_pair(sRing + slot * Cfg::TILE_BYTES + i * 8192, map, full0 + slot * 8, x0 + i * dx, y0 + i * dy, z);
        if (++slot == base + n) { slot = base; ph ^= 1; }
        s_issued[is_s ? 0 : 1] = ++id;
      };
      for (int kb = 0; kb < nkb && ok; ++kb) {
        if (is_s) {
          for (int a = 0; a < cq && ok; ++a) put(&tmKt, 0, 64, kb * BC + (int)rank * 64, 0, bh * cq + a);
          if (ok) put(&tmV, 0, 64, kb * BC + (int)rank * 64, 0, bh);
        } else {
          for (int a = 0; a < cq && ok; ++a) put(&tmKd, (int)rank * (D / 2), 0, kb * BC, 64, bh * cq + a);
        }
      }
      // the last arrivals on this CTA's `empty` barriers have landed before it leaves
      for (int i = 0; i < n && i < id && ok; ++i) {
        if (--slot < base) { slot = base + n - 1; ph ^= 1; }
        ok = tc::mbar_wait(&empty[slot], ph ^ 1, s_abort);
      }
    }
  } else if (role == 1 || role == 3) {
    // ===================== MMA issuers (rank 0) =====================
    if (nkb > 0 && rank == 0) {   // all lanes run the loop; one elected lane issues
      constexpr uint32_t idescS = tc::make_idesc(2 * BM, BC, 0, 0);    // S, dP: both operands K-major
      constexpr uint32_t idescQ = tc::make_idesc(2 * BM, D, 0, 1);     // dQ: B (Kt) MN-major
      const uint64_t d128 = tc::make_sdesc(smem_u32(sRing), 16, 1024, tc::kLayoutSW128);
      const uint64_t d64 = tc::make_sdesc(smem_u32(sRing), 16, 512, tc::kLayoutSW64);
      const uint32_t hi = (uint32_t)(d128 >> 32), r_lo = (uint32_t)d128, d_hi = D == 64 ? (uint32_t)(d64 >> 32) : hi;
      const uint32_t s_lo = r_lo - (uint32_t)(Cfg::oRing >> 4);        // descriptor of shared-memory offset 0
      bool ok = true;
      auto wait = [&](uint64_t* bar, int n) {                          // completion n of the barrier
        ok = tc::mbar_wait_warp(bar, n & 1, s_abort);
        tc::tc_fence_after();
      };
      if (role == 1) {
        const uint32_t q_lo = s_lo + (uint32_t)((Cfg::oQ + (HALO - pq) * 128) >> 4), o_lo = s_lo + (uint32_t)(Cfg::oO >> 4);
        tc::TileRing<NSS> ring(full, empty, s_abort);
        ok = tc::mbar_wait_warp(q_full, 0, s_abort);
        for (int kb = 0; kb < nkb && ok; ++kb) {
          if (kb > 0) wait(s_free, kb - 1);                              // S(kb-1) has been taken
          for (int a = 0; a < cq && ok; ++a) {
            if (!(ok = ring.take())) break;
#pragma unroll
            for (int sl = 0; sl < SLABS; ++sl)
              tc::mma4_ss<2>(tmem + Cfg::colS, q_lo + (uint32_t)((sl * Cfg::Q_SLAB + a * 128) >> 4), hi, 2,
                             r_lo + (uint32_t)((ring.slot * Cfg::TILE_BYTES + sl * 8192) >> 4), hi, 2, idescS, (a | sl) != 0);
            ring.give();
          }
          if (!ok) break;
          tc::mma_commit_pair(s_full);
          if (kb > 0) wait(p_free, kb - 1);
          if (!ok || !(ok = ring.take())) break;
#pragma unroll
          for (int sl = 0; sl < SLABS; ++sl)
            tc::mma4_ss<2>(tmem + Cfg::colP, o_lo + (uint32_t)((sl * Cfg::O_SLAB) >> 4), hi, 2,
                           r_lo + (uint32_t)((ring.slot * Cfg::TILE_BYTES + sl * 8192) >> 4), hi, 2, idescS, sl != 0);
          ring.give();
          tc::mma_commit_pair(p_full);
        }
      } else {
        const uint32_t c_lo = s_lo + (uint32_t)(Cfg::oC >> 4), rd_lo = r_lo + (uint32_t)(NSS * (Cfg::TILE_BYTES >> 4));
        tc::TileRing<NSLOT - NSS> ring(full + NSS, empty + NSS, s_abort);
        for (int kb = 0; kb < nkb && ok; ++kb) {
          wait(dc_full, kb);
          for (int a = 0; a < cq && ok; ++a) {
            if (!(ok = ring.take())) break;
            const uint32_t b_lo = rd_lo + (uint32_t)(ring.slot * (Cfg::TILE_BYTES >> 4));
            const uint32_t a_lo = c_lo + (uint32_t)(((pq - a) * 128) >> 4);      // dC rows i' + pad_q - a
            constexpr uint32_t step = D == 64 ? 64 : 128;                        // 16 keys
            tc::mma4_ss<2>(tmem + Cfg::colQ, a_lo, hi, 2, b_lo, d_hi, step, idescQ, (kb | a) != 0);
            tc::mma4_ss<2>(tmem + Cfg::colQ, a_lo + (uint32_t)(Cfg::C_SLAB >> 4), hi, 2, b_lo + 4 * step, d_hi, step, idescQ, 1);
            ring.give();
          }
          if (!ok) break;
          tc::mma_commit_pair(dq_done);
        }
      }
    }
  } else {
    // ===================== element-wise warps: one dC row and 64 of the 128 keys per thread =====================
    const int c = warp >> 2;                            // key half
    const int m = (warp & 3) * 32 + lane;               // row within the tile = TMEM lane
    const int gi = R0 + (int)rank * OWN + m;  // query index of this dC row
    const uint32_t tT = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t tS = tT + Cfg::colS + c * 64, tP = tT + Cfg::colP + c * 64, tQ = tT + Cfg::colQ + c * (D / 2);
    const uint32_t r_sfree = tc::cluster_addr(s_free, 0), r_pfree = tc::cluster_addr(p_free, 0), r_dc = tc::cluster_addr(dc_full, 0);
    const bool row_ok = gi >= 0 && gi < N;
    const float lse2 = row_ok ? p.LSE[(size_t)bh * N + gi] * kLog2e : 0.f;
    const float dvec = row_ok ? p.Dvec[(size_t)bh * N + gi] : 0.f;
    const int jlim = row_ok ? (p.causal ? min(N - 1, gi - band) : N - 1) : -1;   // last key owned here
    unsigned char* cbuf = smem + Cfg::oC + c * Cfg::C_SLAB + m * 128;   // 16-byte chunk k of the row at chunk k ^ (row & 7)
    bool ok = true;
    for (int kb = 0; kb < nkb && ok; ++kb) {
      ok = __all_sync(0xffffffffu, (p.selftest_expire && kb == 0)
                                       ? tc::mbar_wait(never_bar, 0, s_abort, tc::kSelfTestSpinLimit)
                                       : tc::mbar_wait(s_full, kb & 1, s_abort));
      if (!ok) break;   // warp-uniform: the TMEM accesses below are warp-collective
      tc::tc_fence_after();
      float s[64];
      tc::tmem_ld32_nowait(tS, reinterpret_cast<float(&)[32]>(s[0]));
      tc::tmem_ld32_nowait(tS + 32, reinterpret_cast<float(&)[32]>(s[32]));
      tc::tmem_wait_ld();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive_cluster(r_sfree);
#pragma unroll
      for (int i = 0; i < 64; ++i) s[i] = exp2f(s[i] - lse2);
      const int j0 = kb * BC + c * 64;
      if (j0 + 63 > jlim) {
#pragma unroll
        for (int i = 0; i < 64; ++i) if (j0 + i > jlim) s[i] = 0.f;
      }
      ok = __all_sync(0xffffffffu, tc::mbar_wait(p_full, kb & 1, s_abort));
      if (!ok) break;
      tc::tc_fence_after();
      uint32_t pk32[32];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float dp[16];
        tc::tmem_ld16(tP + 16 * q, dp);
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const float c0 = s[16 * q + i], c1 = s[16 * q + i + 1];       // 0 where masked, whatever dP is there
          pk32[8 * q + i / 2] = pack_bf16(c0 * (dp[i] - dvec), c1 * (dp[i + 1] - dvec));
        }
      }
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive_cluster(r_pfree);
      if (kb > 0) {   // dQ(kb-1) has finished reading the dC buffer
        ok = __all_sync(0xffffffffu, tc::mbar_wait(dq_done, (kb - 1) & 1, s_abort));
        if (!ok) break;
      }
#pragma unroll
      for (int k = 0; k < 8; ++k)
        *reinterpret_cast<uint4*>(cbuf + ((k ^ (m & 7)) << 4)) = make_uint4(pk32[4 * k], pk32[4 * k + 1], pk32[4 * k + 2], pk32[4 * k + 3]);
      tc::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive_cluster(r_dc);
    }
    // ---- epilogue: the owned dQ rows of this tile, half the columns per thread ----
    if (nkb > 0 && ok) ok = __all_sync(0xffffffffu, tc::mbar_wait(dq_done, (nkb - 1) & 1, s_abort));
    tc::tc_fence_after();
    const bool have = (nkb > 0) && ok;
    const bool store = row_ok && (m < OWN) && (gi >= p.row_base) && (gi < p.row_end);
    const size_t orow = ((size_t)bh * N + (row_ok ? gi : 0)) * D + c * (D / 2);
    if (p.early) pdl_wait();                            // the band kernel's part of dQ
#pragma unroll
    for (int q = 0; q < D / 64; ++q) {
      float o[32];
      if (have) {
        tc::tmem_ld32(tQ + q * 32, o);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = 0.f;
      }
      if (store) store_grad32(p.dQ, p.out_bf16, p.dQadd, orow + q * 32, o, kLn2);
    }
  }
  __syncwarp();

  // ===================== teardown =====================
  if (tid == 0 && *s_abort) tc::st_cluster_u32(tc::cluster_addr((const void*)s_abort, rank ^ 1), 1);
  tc::tc_fence_before();
  tc::cluster_sync_all();
  if (*s_abort) {        // of either CTA
    if (tid == 0) atomicExch(p.status, 1);
    // nothing of the pair may still be in flight when its shared and tensor memory are given up: the issuer commits
    // behind its last MMA, one thread waits (bounded) for that commit and for the copies issued last into each slot
    if (rank == 0 && (role == 1 || role == 3)) tc::mma_commit_pair(mma_drain);
    if (rank == 0 && tid == EW * 32 && nkb > 0) {
      volatile int never = 0;
      constexpr uint32_t kDrain = 1u << 14;
      tc::mbar_wait(q_full, 0, &never, kDrain);
      for (int r = 0; r < 2; ++r) {
        const int issued = s_issued[r], base = r ? NSS : 0, n = r ? NSLOT - NSS : NSS;
        for (int id = max(0, issued - n); id < issued; ++id) tc::mbar_wait(&full[base + id % n], (id / n) & 1, &never, kDrain);
      }
    }
    if (tid == EW * 32) { volatile int never = 0; tc::mbar_wait(mma_drain, 0, &never); }
    tc::cluster_sync_all();
  }
  if (warp == EW + 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc_pair(tmem, Cfg::kTmemCols);
  }
}

namespace {

template <int D>
cudaError_t launch_t(const TrainParams& p, __nv_bfloat16* Kt, int* status, cudaStream_t stream) {
  using Cfg = DqCfg<D>;
  const size_t BH = (size_t)p.B * p.H;
  alignas(64) CUtensorMap tmQ, tmdO, tmKt, tmKd, tmV;
  if (!make_tensor_map_bf16(&tmQ, p.Q, D, p.N, BH, 64, Cfg::BM + Cfg::HALO, true)) return cudaErrorInvalidValue;
  if (!make_tensor_map_bf16(&tmdO, p.dO, D, p.N, BH, 64, Cfg::BM, true)) return cudaErrorInvalidValue;
  if (!make_tensor_map_bf16(&tmKt, Kt, D, p.N, BH * p.cq, 64, 64, true)) return cudaErrorInvalidValue;
  if (!make_tensor_map_bf16(&tmKd, Kt, D, p.N, BH * p.cq, D / 2, D == 64 ? 128 : 64, true)) return cudaErrorInvalidValue;
  if (!make_tensor_map_bf16(&tmV, p.V, D, p.N, BH, 64, 64, true)) return cudaErrorInvalidValue;
  BwdTcParams bp = {};
  bp.LSE = p.LSE; bp.Dvec = p.Dvec; bp.dQ = p.dQo; bp.dQadd = p.causal ? p.dQ : nullptr; bp.out_bf16 = p.grad_bf16; bp.status = status;
  bp.early = p.causal;
  bp.B = p.B; bp.H = p.H; bp.N = p.N; bp.cq = p.cq; bp.ck = p.ck; bp.causal = p.causal;
  bp.selftest_expire = take_selftest_expire(kKernBwdDqTc);
  bp.row_base = win_lo(p); bp.row_end = win_hi(p);
  bp.own = Cfg::BM - (p.cq - 1);
  const int rows = bp.own * 2;
  auto kern = bwd_dq_tc_kernel<D>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
  if (e != cudaSuccess) return e;
  dim3 grid(2u * (unsigned)((bp.row_end - bp.row_base + rows - 1) / rows) * (unsigned)BH);
  ScopedKernelTimer timer_(kKernBwdDqTc, stream);
  return launch_pdl(kern, grid, dim3(Cfg::kThreads), Cfg::kSmemBytes, stream, tmQ, tmdO, tmKt, tmKd, tmV, bp);
}

}  // namespace

cudaError_t launch_bwd_dq_pair(const TrainParams& p, __nv_bfloat16* Kt, int* status, cudaStream_t stream) {
  return p.d == 128 ? launch_t<128>(p, Kt, status, stream) : launch_t<64>(p, Kt, status, stream);
}

}  // namespace fmta

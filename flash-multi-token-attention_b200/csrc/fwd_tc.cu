// Stacked-GEMM conv-attention forward on the 5th-generation tensor cores (tcgen05 + TMEM + TMA).
//
// Off the causal band (query - key >= pad_q + pad_k) the conv'd logits are a plain GEMM with a
// stacked contraction:
//     C[i,j] = sum_a  q_{i-(pad_q-a)} . Kt_a[j],     Kt_a[j] = scale * sum_b theta[a,b] k_{j+b-pad_k}
// so those tiles are FlashAttention with c_q accumulating MMAs per score tile and no work on the
// FP32 pipe.  This file holds
//   ktilde_kernel : the memory-bound pre-pass that writes the c_q bf16 operands Kt_a;
//   fwd_tc_kernel : the warp-specialised main kernel, a cluster of two CTAs (1 TMA warp, 1 MMA warp, 8 softmax warps each);
//   launch_fwd_tc : tensor maps + launches.
// Ownership is per score entry: the stacked kernel takes every entry with query - key >= pad_q +
// pad_k (masking the rest of a diagonal tile), the band kernel (fwd_band.cu) takes the band entries.  The
// kernel leaves an UN-normalised partial (O, m, l) per query row; the band kernel continues the
// online softmax from that state over the band and writes the final O, M, L.
//
// Row-shifted A operands without copies: Q is staged as a 128-byte-swizzled tile; the tensor core applies the swizzle
// to the absolute shared-memory address, so the operand "Q shifted by s rows" is the same buffer with the descriptor
// start address advanced by 128*s bytes.
//
// Every wait on an mbarrier is bounded (tc::mbar_wait); on expiry the CTA raises an abort flag, both CTAs of the pair
// drain their outstanding copies, record it in the caller's status word, free their TMEM and return.  No TMA multicast.
#include <cuda.h>
#include <cuda_runtime.h>

#include <mutex>

#include "fmta_params.h"
#include "fmta_tc.cuh"
#include "launch_util.cuh"

namespace fmta {


// what eight bf16 roundings leave over, as bf16
FMTA_DEVINL uint4 bf16_rest(const float (&v)[8], const uint4& o) {
  const uint32_t h[4] = {o.x, o.y, o.z, o.w};
  uint32_t r[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) r[e] = pack_bf16(v[2 * e] - __uint_as_float(h[e] << 16), v[2 * e + 1] - __uint_as_float(h[e] & 0xffff0000u));
  return make_uint4(r[0], r[1], r[2], r[3]);
}

// ------------------------------------------------------------------------------------------
// Kt[bh, a, j, :] = scale * sum_b theta[h, a, b] * K[bh, j + b - pad_k, :]   (bf16, zero beyond ends)
template <int D, bool LO>   // LO: a (hi, lo) bf16 pair per tap
__global__ void __launch_bounds__(256) ktilde_kernel(const bf16* __restrict__ K, const float* __restrict__ theta,
                                                     bf16* __restrict__ Kt, int H, int N, int cq, int ck,
                                                     float scale) {
  // one thread = one 16-byte chunk of one output row of ONE tap (blockIdx.z): light threads, many of them
  constexpr int CPR = D / 8;          // 16-byte chunks per row
  constexpr int RPB = 256 / CPR;      // rows per block
  __shared__ float sTh[20];
  const int bh = blockIdx.y, h = bh % H, a = blockIdx.z;
  pdl_trigger();
  pdl_wait();      // before any read: the kernel in front may have written K or the filter (an optimizer, a cast)
  if (threadIdx.x < ck) sTh[threadIdx.x] = theta[((size_t)h * cq + a) * ck + threadIdx.x] * scale;   // scale carries log2(e)
  __syncthreads();
  const int j = blockIdx.x * RPB + threadIdx.x / CPR, c = threadIdx.x % CPR;
  if (j >= N) return;
  const int pk = (ck - 1) / 2;
  const bf16* Kb = K + (size_t)bh * N * D + c * 8;
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.f;
#pragma unroll 4
  for (int b = 0; b < ck; ++b) {
    const int jj = j + b - pk;
    if (jj < 0 || jj >= N) continue;
    const uint4 kv = *reinterpret_cast<const uint4*>(Kb + (size_t)jj * D);
    const float w = sTh[b];
    const uint32_t w32[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      acc[2 * e] = fmaf(w, __uint_as_float(w32[e] << 16), acc[2 * e]);
      acc[2 * e + 1] = fmaf(w, __uint_as_float(w32[e] & 0xffff0000u), acc[2 * e + 1]);
    }
  }
  uint4 o;
  o.x = pack_bf16(acc[0], acc[1]); o.y = pack_bf16(acc[2], acc[3]);
  o.z = pack_bf16(acc[4], acc[5]); o.w = pack_bf16(acc[6], acc[7]);
  bf16* dst = Kt + ((((size_t)bh * cq + a) * (LO ? 2 : 1)) * N + j) * D + c * 8;
  *reinterpret_cast<uint4*>(dst) = o;
  if (LO) *reinterpret_cast<uint4*>(dst + (size_t)N * D) = bf16_rest(acc, o);
}

// Same pre-pass with the filter width known at compile time: one thread owns one 16-byte column
// chunk of RR consecutive rows and produces all c_q taps from a register window of RR + CK - 1
// key rows, so every key row is loaded once per RR outputs instead of once per output and tap.
template <int D, int CK, int RR, bool LO>
__global__ void __launch_bounds__(256) ktilde_window_kernel(const bf16* __restrict__ K, const float* __restrict__ theta,
                                                            bf16* __restrict__ Kt, int H, int N, int cq, float scale) {
  constexpr int CPR = D / 8, RUNS = 256 / CPR, PK = (CK - 1) / 2, WIN = RR + CK - 1;
  __shared__ float sTh[16 * CK];
  const int bh = blockIdx.y, h = bh % H;
  pdl_trigger();
  pdl_wait();      // before any read: the kernel in front may have written K or the filter (an optimizer, a cast)
  const int j0 = (blockIdx.x * RUNS + threadIdx.x / CPR) * RR, c = threadIdx.x % CPR;
  const bf16* Kb = K + (size_t)bh * N * D + c * 8;
  uint4 win[WIN];
#pragma unroll
  for (int r = 0; r < WIN; ++r) {
    const int jj = j0 + r - PK;
    win[r] = (jj >= 0 && jj < N) ? *reinterpret_cast<const uint4*>(Kb + (size_t)jj * D) : make_uint4(0u, 0u, 0u, 0u);
  }
  for (int i = threadIdx.x; i < cq * CK; i += 256) sTh[i] = theta[(size_t)h * cq * CK + i] * scale;
  __syncthreads();
  if (j0 >= N) return;
  for (int a = 0; a < cq; ++a) {
    float w[CK];
#pragma unroll
    for (int b = 0; b < CK; ++b) w[b] = sTh[a * CK + b];
    bf16* out = Kt + ((((size_t)bh * cq + a) * (LO ? 2 : 1)) * N + j0) * D + c * 8;
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      float acc[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = 0.f;
#pragma unroll
      for (int b = 0; b < CK; ++b) {
        const uint4 kv = win[r + b];
        const uint32_t w32[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          acc[2 * e] = fmaf(w[b], __uint_as_float(w32[e] << 16), acc[2 * e]);
          acc[2 * e + 1] = fmaf(w[b], __uint_as_float(w32[e] & 0xffff0000u), acc[2 * e + 1]);
        }
      }
      if (j0 + r < N) {
        uint4 o;
        o.x = pack_bf16(acc[0], acc[1]); o.y = pack_bf16(acc[2], acc[3]);
        o.z = pack_bf16(acc[4], acc[5]); o.w = pack_bf16(acc[6], acc[7]);
        *reinterpret_cast<uint4*>(out + (size_t)r * D) = o;
        if (LO) *reinterpret_cast<uint4*>(out + (size_t)(N + r) * D) = bf16_rest(acc, o);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------
struct TcParams {
  float* Opart;   // [B,H,N,D] un-normalised
  float* Mpart;   // [B,H,N]  row max, natural-log units
  float* Lpart;
  int* status;    // device word: set non-zero when a bounded wait expired
  int B, H, N, cq, ck, causal;
  int qb_lo, qb_hi;      // row blocks [qb_lo, qb_hi) of 256 rows (all of them unless the call has a window)
  int selftest_expire;   // failure-detection self-test: the softmax warps' first wait is on a barrier nothing arrives at
};

// Two CTAs own 256 query rows (128 each: one TMEM lane per row) and walk blocks of 128 keys.
//   S = sum_a Q^(a) Kt_a^T : 256 x 128 x 16 MMAs, each CTA stages its own Q and HALF the keys of every Kt tile;
//   O += P V               : 256 x d x 16 MMAs, P in tensor memory, each CTA stages half the columns of V.
// A single CTA's 128 x 128 x 16 MMA reads 8 KB of operands in 64 cycles, all the shared memory can deliver; a pair's reads
// 6 KB per CTA, which leaves room for the copies that fill the ring, and every key tile crosses from L2 once for 256 rows.
//   d = 64 : 256 tensor-memory columns and 113 KB, so two pairs share two SMs: one's softmax under the other's MMAs;
//   d = 128: S is double-buffered instead (2 x 128 + 64 + 128 columns).
// Measured (B200, c_q 6, causal, N 4096, single CTAs with two row tiles before): d = 64, B 4, H 16: 415 -> 370 us; d = 128,
// B 8, H 32: 4.33 -> 3.7 ms (1040 TFLOP/s); one sequence of N 1000, 8 heads, d = 128: 80 -> 45 us with the pre-pass and the
// band kernel.  What bounds it is the supply of key tiles (31 bytes per cycle and SM at the tensor core's rate) and power.
template <int D>
struct TcCfg {
  static constexpr int BM = 128, BC = 128;
  static constexpr int HALO = 16;              // rows staged above the block (pad_q <= 15)
  static constexpr int QR = BM + HALO;
  static constexpr int SLABS = D / 64;         // 64-element (128-byte) column slabs per row
  static constexpr int VW = D / 2;             // V columns staged by one CTA
  static constexpr int VT = (BC * VW * 2) / 8192;   // ring tiles of one V half: 1 (d = 64: 128 keys x 32, 64-byte swizzle) or 2 (64 keys x 64)
  static constexpr int TILE_BYTES = 8192;      // Kt: 64 keys x 64 elements, 128-byte swizzle
  static constexpr int NS = (D == 64) ? 1 : 2; // S buffers
  static constexpr int NSLOT = (D == 64) ? 11 : 23;   // d = 64: two CTAs share an SM
  static constexpr int oQ = 0;                 // [d/64][QR][128 B], 128-byte swizzle
  static constexpr int oRing = ((oQ + QR * D * 2 + 1023) / 1024) * 1024;
  static constexpr int oMax = oRing + NSLOT * TILE_BYTES;    // row maxima, exchanged between the two column halves: [2][2][128]
  static constexpr int oBar = oMax + 2 * 2 * BM * 4;
  static constexpr int kSmemBytes = oBar + 512 + 1024;       // + alignment slack
  static constexpr int colS = 0, colP = NS * BC, colO = colP + BC / 2;
  static constexpr int kTmemCols = (D == 64) ? 256 : 512;
  static constexpr int kEw = 8;                // softmax warps: 4 lane quarters x 2 column halves
  static constexpr int kThreads = (kEw + 2) * 32;
  static_assert(colO + D <= kTmemCols, "TMEM budget");
  static_assert(kSmemBytes <= (D == 64 ? 113 : 227) * 1024, "shared memory budget");
};

constexpr float kRescaleTau = 8.f;   // log2 units: P may reach 2^8 before O is rescaled

template <int D>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TcCfg<D>::kThreads, D == 64 ? 2 : 1)
fwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKt,
                const __grid_constant__ CUtensorMap tmV, const TcParams p) {
  using Cfg = TcCfg<D>;
  constexpr int BM = Cfg::BM, BC = Cfg::BC, HALO = Cfg::HALO, QR = Cfg::QR, NSLOT = Cfg::NSLOT, NS = Cfg::NS;
  constexpr int SLABS = Cfg::SLABS, EW = Cfg::kEw;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* sQ = smem + Cfg::oQ;
  unsigned char* sRing = smem + Cfg::oRing;
  float* sMax = reinterpret_cast<float*>(smem + Cfg::oMax);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::oBar);
  // (rank 0): only the copy in rank 0's shared memory is used
  uint64_t* full = bars;                 // [NSLOT]  TMA of both CTAs -> MMA (rank 0)
  uint64_t* empty = bars + NSLOT;        // [NSLOT]  MMA -> TMA
  uint64_t* q_full = bars + 2 * NSLOT;   // (rank 0)
  uint64_t* s_full = q_full + 1;         // [NS]  S ready
  uint64_t* s_free = s_full + NS;        // [NS]  S loaded into registers by all warps of both CTAs (rank 0)
  uint64_t* p_full = s_free + NS;        // P written to tensor memory (rank 0)
  uint64_t* o_full = p_full + 1;         // PV(kb) completed
  uint64_t* xch = o_full + 1;            // [4]  both warps of 32 rows have left their maxima in shared memory
  uint64_t* never_bar = xch + 4;         // nothing arrives here (expiry self-test)
  uint64_t* mma_drain = never_bar + 1;   // abort path: the issued MMAs have completed
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(mma_drain + 1);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
  volatile int* s_issued = s_abort + 1;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = tc::cluster_rank();
  const int N = p.N, cq = p.cq, pq = cq - 1, pk = (p.ck - 1) / 2;
  const int band = pq + pk;              // entries with query - key < band belong to the band kernel
  int bh, qb;
  tc::pair_block_order(blockIdx.x >> 1, p.qb_hi - p.qb_lo, p.B * p.H, bh, qb);
  qb = p.qb_hi - 1 - qb;
  const int P0 = qb * 2 * BM, i0 = P0 + (int)rank * BM;     // first row of the pair, of this CTA
  int nkb = (N + BC - 1) / BC;
  if (p.causal) {                        // key blocks that hold at least one key j <= (last row) - band
    const int last = min(N - 1, P0 + 2 * BM - 1) - band;
    nkb = last >= 0 ? min(nkb, last / BC + 1) : 0;
  }

  if (tid == 0) {
    for (int i = 0; i < NSLOT; ++i) { tc::mbar_init(&full[i], 1); tc::mbar_init(&empty[i], 1); }
    tc::mbar_init(q_full, 1);
    for (int i = 0; i < NS; ++i) { tc::mbar_init(&s_full[i], 1); tc::mbar_init(&s_free[i], 2 * EW); }
    tc::mbar_init(p_full, 2 * EW); tc::mbar_init(o_full, 1);
    for (int i = 0; i < 4; ++i) tc::mbar_init(&xch[i], 2);
    tc::mbar_init(never_bar, 1); tc::mbar_init(mma_drain, 1);
    *s_abort = 0; *s_issued = 0;
    tc::mbar_fence_init();
  }
  if (warp == EW + 1) tc::tmem_alloc_pair(s_tmem, Cfg::kTmemCols);
  tc::tc_fence_before();
  tc::cluster_sync_all();
  pdl_wait();      // nothing before this line touches global memory that a kernel of this library writes or reads back
  pdl_trigger();   // after the wait: the band kernel behind this one reads Q, K, V before it waits for this kernel
  tc::tc_fence_after();
  const uint32_t tmem = *s_tmem;

  if (warp == EW) {
    // ===================== TMA producer: this CTA's Q, its half of every Kt and V tile =====================
    if (lane == 0 && nkb > 0) {
      tc::tma_prefetch_desc(&tmQ); tc::tma_prefetch_desc(&tmKt); tc::tma_prefetch_desc(&tmV);
      const uint32_t full0 = tc::cluster_addr(full, 0);
      if (rank == 0) tc::mbar_expect_tx(q_full, 2 * QR * D * 2);
      const uint32_t qf = tc::cluster_addr(q_full, 0);
      for (int sl = 0; sl < SLABS; ++sl) tc::tma_load_3d_pair(sQ + sl * (QR * 128), &tmQ, qf, sl * 64, i0 - HALO, bh);
      int slot = 0, ph = 1, id = 0;
      bool ok = true;
      auto put = [&](const CUtensorMap* map, int x, int y, int z) {
        if (!tc::mbar_wait(&empty[slot], ph, s_abort)) { ok = false; return; }
        if (rank == 0) tc::mbar_expect_tx(&full[slot], 2 * Cfg::TILE_BYTES);
        tc::tma_load_3d_pair(sRing + slot * Cfg::TILE_BYTES, map, full0 + slot * 8, x, y, z);
        if (++slot == NSLOT) { slot = 0; ph ^= 1; }
        *s_issued = ++id;
      };
      auto put_K = [&](int kb) {
        for (int a = 0; a < cq && ok; ++a)
          for (int sl = 0; sl < SLABS && ok; ++sl) put(&tmKt, sl * 64, kb * BC + (int)rank * (BC / 2), bh * cq + a);
      };
      // same order as the MMA warp consumes: S(0); then S(kb+1), V(kb)
      put_K(0);
      for (int kb = 0; kb < nkb && ok; ++kb) {
        if (kb + 1 < nkb) put_K(kb + 1);
        for (int v = 0; v < Cfg::VT && ok; ++v) put(&tmV, (int)rank * Cfg::VW, kb * BC + v * 64, bh);
      }
      // the last arrivals on this CTA's `empty` barriers have landed before it leaves
      for (int i = 0; i < NSLOT && i < id && ok; ++i) {
        if (--slot < 0) { slot = NSLOT - 1; ph ^= 1; }
        ok = tc::mbar_wait(&empty[slot], ph ^ 1, s_abort);
      }
    }
  } else if (warp == EW + 1) {
    // ===================== MMA issuer (rank 0) =====================
    if (nkb > 0 && rank == 0) {   // all lanes run the loop; one elected lane issues (see tc::elect_one)
      constexpr uint32_t idescS = tc::make_idesc(2 * BM, BC, 0, 0);
      constexpr uint32_t idescPV = tc::make_idesc(2 * BM, D, 0, 1);
      // descriptors split into a constant high word and a low word that carries the start address
      // row shift: the same tile with the start address moved by 128 bytes per row (the tensor core applies the
      // swizzle to the absolute shared-memory address, as TMA did)
      const uint64_t dQ0 = tc::make_sdesc(smem_u32(sQ) + (HALO - pq) * 128, 16, 1024, tc::kLayoutSW128);
      const uint64_t dK0 = tc::make_sdesc(smem_u32(sRing), 16, 1024, tc::kLayoutSW128);
      const uint64_t dV0 = D == 64 ? tc::make_sdesc(smem_u32(sRing), 16, 512, tc::kLayoutSW64) : dK0;
      const uint32_t a_hi = (uint32_t)(dQ0 >> 32), a_lo0 = (uint32_t)dQ0;
      const uint32_t k_hi = (uint32_t)(dK0 >> 32), v_hi = (uint32_t)(dV0 >> 32), b_lo0 = (uint32_t)dK0;
      tc::TileRing<NSLOT> ring(full, empty, s_abort);
      bool ok = tc::mbar_wait_warp(q_full, 0, s_abort);
      auto issue_S = [&](int kb) {
        const int buf = kb % NS;
        const uint32_t dS = tmem + Cfg::colS + buf * BC;
        if (kb >= NS) {      // the softmax threads have taken block kb - NS out of this buffer
          ok = tc::mbar_wait_warp(&s_free[buf], (kb / NS - 1) & 1, s_abort);
          if (!ok) return;
          tc::tc_fence_after();
        }
        uint32_t a_lo = a_lo0;
        for (int a = 0; a < cq; ++a, a_lo += 128 >> 4) {
#pragma unroll
          for (int sl = 0; sl < SLABS; ++sl) {
            if (!(ok = ring.take())) return;
            const uint32_t b_lo = b_lo0 + (uint32_t)(ring.slot * (Cfg::TILE_BYTES >> 4));
            tc::mma4_ss<2>(dS, a_lo + (uint32_t)(sl * (QR * 128 >> 4)), a_hi, 2, b_lo, k_hi, 2, idescS, (a | sl) != 0);
            ring.give();
          }
        }
        tc::mma_commit_pair(&s_full[buf]);
      };
      auto issue_PV = [&](int kb) {
        ok = tc::mbar_wait_warp(p_full, kb & 1, s_abort);
        if (!ok) return;
#pragma unroll
        for (int v = 0; v < Cfg::VT; ++v) {
          if (!(ok = ring.take())) return;
          const uint32_t b_lo = b_lo0 + (uint32_t)(ring.slot * (Cfg::TILE_BYTES >> 4));
#pragma unroll
          for (int k = 0; k < BC / 16 / Cfg::VT; k += 4)       // 16 keys: 16 rows of V, 8 columns of P
            tc::mma4_ts<2>(tmem + Cfg::colO, tmem + Cfg::colP + 8 * (v * 4 + k), 8, b_lo + (uint32_t)(k * (16 * Cfg::VW * 2 / 16)), v_hi,
                           16 * Cfg::VW * 2 / 16, idescPV, (kb | v | k) != 0);
          ring.give();
        }
        tc::mma_commit_pair(o_full);
      };
      if (ok) issue_S(0);
      for (int kb = 0; kb < nkb && ok; ++kb) {
        if (kb + 1 < nkb) issue_S(kb + 1);
        if (ok) issue_PV(kb);
      }
    }
  } else {
    // ===================== softmax warps: one query row and 64 of the 128 keys per thread =====================
    const int c = warp >> 2;                            // column half
    const int m = (warp & 3) * 32 + lane;               // row within the tile = TMEM lane
    const int gi = i0 + m;                              // query index
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + Cfg::colS + c * (BC / 2) + lane_base;
    const uint32_t tP = tmem + Cfg::colP + c * (BC / 4) + lane_base;
    const uint32_t tO = tmem + Cfg::colO + c * (D / 2) + lane_base;
    const uint32_t r_sfree = tc::cluster_addr(s_free, 0), r_pfull = tc::cluster_addr(p_full, 0);
    const int jlim = p.causal ? min(N - 1, gi - band) : N - 1;   // last key this row may see here
    float m_run = -INFINITY, l_run = 0.f;               // log2 units (Kt carries scale * log2(e))
    float m_true = -INFINITY;                           // true row max (m_run lags it by up to tau)
    bool ok = true;
    for (int kb = 0; kb < nkb && ok; ++kb) {
      const int buf = kb % NS;
      ok = __all_sync(0xffffffffu, (p.selftest_expire && kb == 0)
                                       ? tc::mbar_wait(never_bar, 0, s_abort, tc::kSelfTestSpinLimit)
                                       : tc::mbar_wait(&s_full[buf], (kb / NS) & 1, s_abort));
      if (!ok) break;   // warp-uniform: the TMEM accesses below are warp-collective
      tc::tc_fence_after();
      float s[64];
      tc::tmem_ld32_nowait(tS + buf * BC, reinterpret_cast<float(&)[32]>(s[0]));
      tc::tmem_ld32_nowait(tS + buf * BC + 32, reinterpret_cast<float(&)[32]>(s[32]));
      tc::tmem_wait_ld();
      // S is in registers: the MMA warp may overwrite it
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive_cluster(r_sfree + buf * 8);
      const int j0 = kb * BC + c * 64;
      // mask: keys past N, and (causal) entries on or above the band, which the band kernel owns
      if (j0 + 63 > jlim) {
#pragma unroll
        for (int i = 0; i < 64; ++i) if (j0 + i > jlim) s[i] = -INFINITY;
      }
      float mx0 = fmaxf(s[0], s[1]), mx1 = fmaxf(s[2], s[3]), mx2 = fmaxf(s[4], s[5]), mx3 = fmaxf(s[6], s[7]);
#pragma unroll
      for (int i = 8; i < 64; i += 8) {
        mx0 = fmaxf(mx0, fmaxf(s[i], s[i + 1])); mx1 = fmaxf(mx1, fmaxf(s[i + 2], s[i + 3]));
        mx2 = fmaxf(mx2, fmaxf(s[i + 4], s[i + 5])); mx3 = fmaxf(mx3, fmaxf(s[i + 6], s[i + 7]));
      }
      float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
      // both halves of a row use one reference: exchange the maxima (double-buffered: a buffer is rewritten two blocks
      // later, behind the barrier of the block between)
      float* mrow = sMax + (kb & 1) * (2 * BM) + m;
      mrow[c * BM] = mx;
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&xch[warp & 3]);
      ok = __all_sync(0xffffffffu, tc::mbar_wait(&xch[warp & 3], kb & 1, s_abort));
      if (!ok) break;
      mx = fmaxf(mx, mrow[(c ^ 1) * BM]);
      m_true = fmaxf(m_true, mx);
      // lazy rescale: keep the reference max until a block exceeds it by more than tau
      float alpha = 1.f;
      bool need = false;
      if (m_run == -INFINITY) {
        m_run = mx;                                     // O and l are still zero: nothing to rescale
      } else if (mx > m_run + kRescaleTau) {
        alpha = exp2f(m_run - mx);
        m_run = mx;
        need = true;
      }
      const float mref = (m_run == -INFINITY) ? 0.f : m_run;
      float sum0 = 0.f, sum1 = 0.f;
      uint32_t pk32[32];
#pragma unroll
      for (int i = 0; i < 64; i += 4) {
        const float p0 = exp2f(s[i] - mref), p1 = exp2f(s[i + 1] - mref);
        const float p2 = exp2f(s[i + 2] - mref), p3 = exp2f(s[i + 3] - mref);
        sum0 += p0 + p1; sum1 += p2 + p3;
        pk32[i / 2] = pack_bf16(p0, p1); pk32[i / 2 + 1] = pack_bf16(p2, p3);
      }
      l_run = l_run * alpha + (sum0 + sum1);
      if (kb > 0) {
        // PV(kb-1) complete: P may be overwritten and O touched.  Waited for on every block
        // (not only when O is rescaled) so that the parity wait never aliases an older phase.
        ok = __all_sync(0xffffffffu, tc::mbar_wait(o_full, (kb - 1) & 1, s_abort));
        if (!ok) break;
        tc::tc_fence_after();
      }
      if (__any_sync(0xffffffffu, need)) {   // O *= alpha (need is false on the first block)
#pragma unroll
        for (int q = 0; q < D / 64; ++q) {
          float o[32];
          tc::tmem_ld32(tO + q * 32, o);
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] *= alpha;
          tc::tmem_st32(tO + q * 32, o);
        }
      }
      tc::tmem_st32u(tP, pk32);
      tc::tmem_wait_st();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive_cluster(r_pfull);
    }
    // ---- epilogue: un-normalised partial row ----
    if (nkb > 0 && ok) ok = __all_sync(0xffffffffu, tc::mbar_wait(o_full, (nkb - 1) & 1, s_abort));
    tc::tc_fence_after();
    if (ok) {                                           // row sum: the two halves together
      float* lrow = sMax + (nkb & 1) * (2 * BM) + m;
      lrow[c * BM] = l_run;
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&xch[warp & 3]);
      ok = __all_sync(0xffffffffu, tc::mbar_wait(&xch[warp & 3], nkb & 1, s_abort));
      if (ok) l_run += lrow[(c ^ 1) * BM];
    }
    const bool have = (nkb > 0) && ok;                  // warp-uniform
    // re-reference the partial to the true row max (what the reference reports as M)
    const float fix = (m_true == -INFINITY) ? 0.f : exp2f(m_run - m_true);
    float* orow = p.Opart + ((size_t)bh * N + (gi < N ? gi : 0)) * D + c * (D / 2);
#pragma unroll
    for (int q = 0; q < D / 64; ++q) {
      float o[32];
      if (have) {
        tc::tmem_ld32(tO + q * 32, o);                  // warp-collective: every lane takes part
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = 0.f;
      }
      if (gi < N) {
#pragma unroll
        for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(orow + q * 32 + i) = make_float4(o[i] * fix, o[i + 1] * fix, o[i + 2] * fix, o[i + 3] * fix);
      }
    }
    if (gi < N && c == 0) {
      const bool any = have && (m_run != -INFINITY);
      p.Mpart[(size_t)bh * N + gi] = any ? m_true * 0.6931471805599453f : -INFINITY;
      p.Lpart[(size_t)bh * N + gi] = any ? l_run * fix : 0.f;
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
    if (rank == 0 && warp == EW + 1) tc::mma_commit_pair(mma_drain);
    if (rank == 0 && tid == EW * 32 && nkb > 0) {
      volatile int never = 0;
      constexpr uint32_t kDrain = 1u << 14;
      tc::mbar_wait(q_full, 0, &never, kDrain);
      const int issued = *s_issued;
      for (int id = max(0, issued - NSLOT); id < issued; ++id) tc::mbar_wait(&full[id % NSLOT], (id / NSLOT) & 1, &never, kDrain);
    }
    if (tid == EW * 32) { volatile int never = 0; tc::mbar_wait(mma_drain, 0, &never); }
    tc::cluster_sync_all();
  }
  if (warp == EW + 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc_pair(tmem, Cfg::kTmemCols);
  }
}

// ------------------------------------------------------------------------------------------
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

// cuTensorMapEncodeTiled wants a current context, which a thread gets with its first runtime call that needs one: a thread
// whose first call of this library comes to a kernel without a pre-pass has none yet, and the driver crashes there.
bool context_current() {
  typedef CUresult (*GetCurrentFn)(CUcontext*);
  static const GetCurrentFn fn = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    return cudaGetDriverEntryPoint("cuCtxGetCurrent", &ptr, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess
               ? reinterpret_cast<GetCurrentFn>(ptr) : nullptr;
  }();
  CUcontext ctx = nullptr;
  if (fn && fn(&ctx) == CUDA_SUCCESS && ctx) return true;
  int dev = -1;
  return cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess;
}
}  // namespace

bool tensor_maps_available() { return get_encode_fn() != nullptr; }

// bf16 tensor viewed as [outer][rows][D] (D contiguous); box = {box_x, box_rows, box_outer}
bool make_tensor_map_bf16(CUtensorMap* map, const void* base, int D, int rows, size_t outer, int box_x, int box_rows, bool sw128, int box_outer = 1) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn || !context_current()) return false;
  cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)rows, (cuuint64_t)outer};
  cuuint64_t strides[2] = {(cuuint64_t)D * 2, (cuuint64_t)rows * D * 2};
  cuuint32_t box[3] = {(cuuint32_t)box_x, (cuuint32_t)box_rows, (cuuint32_t)box_outer};
  cuuint32_t es[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, !sw128 ? CU_TENSOR_MAP_SWIZZLE_NONE : box_x == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// fp32 tensor viewed as [outer][rows][D] (D contiguous); box = {box_x, box_rows, 1}; box_x * 4 <= 128 with the swizzle
bool make_tensor_map_f32(CUtensorMap* map, const void* base, int D, int rows, size_t outer, int box_x, int box_rows, bool sw128) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn || !context_current()) return false;
  cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)rows, (cuuint64_t)outer};
  cuuint64_t strides[2] = {(cuuint64_t)D * 4, (cuuint64_t)rows * D * 4};
  cuuint32_t box[3] = {(cuuint32_t)box_x, (cuuint32_t)box_rows, 1};
  cuuint32_t es[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, sw128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Pre-pass: Kt = scale * log2(e) * (theta applied along the key axis of K), c_q bf16 copies.
cudaError_t launch_ktilde(const TrainParams& p, __nv_bfloat16* Kt, cudaStream_t stream, bool with_lo) {
  ScopedKernelTimer timer_(kKernKtilde, stream);
  const size_t BH = (size_t)p.B * p.H;
  const float sc = p.scale * kLog2e;
  if ((p.ck == 11 || p.ck == 9 || p.ck == 7 || p.ck == 5 || p.ck == 3) && p.cq <= 16) {      // filter widths with a register-window instantiation
    constexpr int RR = 4;
#define FMTA_KT_WIN(DD, CKK)                                                                                      \
    { constexpr int RUNS = 256 / (DD / 8);                                                                        \
      dim3 grid((p.N + RUNS * RR - 1) / (RUNS * RR), (unsigned)BH);                                               \
      auto kern = with_lo ? ktilde_window_kernel<DD, CKK, RR, true> : ktilde_window_kernel<DD, CKK, RR, false>;          \
      (void)launch_pdl(kern, grid, dim3(256), 0, stream, p.K, p.theta, Kt, p.H, p.N, p.cq, sc); }
    if (p.d == 64) {
      if (p.ck == 11) FMTA_KT_WIN(64, 11) else if (p.ck == 9) FMTA_KT_WIN(64, 9) else if (p.ck == 7) FMTA_KT_WIN(64, 7) else if (p.ck == 5) FMTA_KT_WIN(64, 5) else FMTA_KT_WIN(64, 3)
    } else {
      if (p.ck == 11) FMTA_KT_WIN(128, 11) else if (p.ck == 9) FMTA_KT_WIN(128, 9) else if (p.ck == 7) FMTA_KT_WIN(128, 7) else if (p.ck == 5) FMTA_KT_WIN(128, 5) else FMTA_KT_WIN(128, 3)
    }
#undef FMTA_KT_WIN
    return cudaGetLastError();
  }
  if (p.d == 64) {
    constexpr int RPB = 256 / (64 / 8);
    dim3 grid((p.N + RPB - 1) / RPB, (unsigned)BH, p.cq);
    return launch_pdl(with_lo ? ktilde_kernel<64, true> : ktilde_kernel<64, false>, grid, dim3(256), 0, stream, p.K, p.theta, Kt, p.H, p.N, p.cq, p.ck, sc);
  } else {
    constexpr int RPB = 256 / (128 / 8);
    dim3 grid((p.N + RPB - 1) / RPB, (unsigned)BH, p.cq);
    return launch_pdl(with_lo ? ktilde_kernel<128, true> : ktilde_kernel<128, false>, grid, dim3(256), 0, stream, p.K, p.theta, Kt, p.H, p.N, p.cq, p.ck, sc);
  }
  return cudaGetLastError();
}

namespace {

template <int D>
cudaError_t launch_tc(const TrainParams& p, bf16* Kt, float* Opart, float* Mpart, float* Lpart, int* status, cudaStream_t stream) {
  using Cfg = TcCfg<D>;
  const size_t BH = (size_t)p.B * p.H;
  alignas(64) CUtensorMap tmQ, tmKt, tmV;
  if (!make_tensor_map_bf16(&tmQ, p.Q, D, p.N, BH, 64, Cfg::QR, true)) return cudaErrorInvalidValue;
  if (!make_tensor_map_bf16(&tmKt, Kt, D, p.N, BH * p.cq, 64, 64, true)) return cudaErrorInvalidValue;
  if (!make_tensor_map_bf16(&tmV, p.V, D, p.N, BH, Cfg::VW, D == 64 ? 128 : 64, true)) return cudaErrorInvalidValue;
  TcParams tp;
  tp.Opart = Opart; tp.Mpart = Mpart; tp.Lpart = Lpart; tp.status = status;
  tp.B = p.B; tp.H = p.H; tp.N = p.N; tp.cq = p.cq; tp.ck = p.ck; tp.causal = p.causal;
  tp.selftest_expire = take_selftest_expire(kKernFwdTc);
  auto kern = fwd_tc_kernel<D>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
  if (e != cudaSuccess) return e;
  constexpr int RB = 2 * Cfg::BM;                                 // rows per pair; a window starts on a multiple of it
  tp.qb_hi = (win_hi(p) + RB - 1) / RB; tp.qb_lo = win_lo(p) / RB;
  dim3 grid(2 * (tp.qb_hi - tp.qb_lo) * (unsigned)BH);
  ScopedKernelTimer timer_(kKernFwdTc, stream);
  return launch_pdl(kern, grid, dim3(Cfg::kThreads), Cfg::kSmemBytes, stream, tmQ, tmKt, tmV, tp);
}

}  // namespace

bool fwd_tc_supported(const TrainParams& p) {
  return p.theta != nullptr && p.Wmix == nullptr && (p.d == 64 || p.d == 128) && p.cq >= 1 && p.cq <= 16 &&
         get_encode_fn() != nullptr;
}

size_t fwd_tc_workspace_bytes(int B, int H, int N, int d, int cq) {
  const size_t rows = (size_t)B * H * N;
  auto up = [](size_t x) { return (x + 1023) / 1024 * 1024; };
  return up(rows * cq * d * 2) + up(rows * d * 4) + 2 * up(rows * 4) + 1024;
}

// Runs the pre-pass and the stacked kernel; on return p_out describes where the band kernel
// must pick up (Opart / Mpart / Lpart).
cudaError_t launch_fwd_tc(const TrainParams& p, void* workspace, const float** Opart, const float** Mpart,
                          const float** Lpart, cudaStream_t stream) {
  const size_t rows = (size_t)p.B * p.H * p.N;
  auto up = [](size_t x) { return (x + 1023) / 1024 * 1024; };
  unsigned char* w = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(workspace) + 1023) & ~uintptr_t(1023));
  bf16* Kt = reinterpret_cast<bf16*>(w); w += up(rows * p.cq * p.d * 2);
  if (p.Kt_ext) Kt = p.Kt_ext;                      // the caller keeps the stacked key operand (for the backward)
  float* Op = reinterpret_cast<float*>(w); w += up(rows * p.d * 4);
  float* Mp = reinterpret_cast<float*>(w); w += up(rows * 4);
  float* Lp = reinterpret_cast<float*>(w); w += up(rows * 4);
  int* status = nullptr;
  cudaError_t e = status_word_of(reinterpret_cast<int*>(w), stream, &status);
  if (e != cudaSuccess) return e;
  if (!(p.Kt_ext && p.kt_valid)) {
    e = launch_ktilde(p, Kt, stream);
    if (e != cudaSuccess) return e;
  }
  e = p.d == 64 ? launch_tc<64>(p, Kt, Op, Mp, Lp, status, stream) : launch_tc<128>(p, Kt, Op, Mp, Lp, status, stream);
  *Opart = Op; *Mpart = Mp; *Lpart = Lp;
  return e;
}


}  // namespace fmta

// Decode (fwd_inference) kernel: last-query-row conv attention over a KV cache, split-K.
//
// Memory-bound: K and V are each read once from HBM with 32-byte loads (16 at d = 32) straight into registers (no shared-memory
// staging, no block-level barrier in the key loop).  Every warp owns a contiguous key range of its split and keeps its own
// online-softmax state; a step is 32 keys:
//   S_a[j] = scale * q_a . k_j for the <= 16 most recent query rows                                   (mma.sync)
//            -> fp32 ring buffer in shared memory (per warp, 64 keys deep)
//   C[j]  = sum_{a,b} theta[a,b] S_a[j+b-pad_k] of the step before, once the first half of this step's scores is there
//            (FP32 pipe; lane = 4 keys x 2 or 4 rows: a window of float4 loads and the filter in registers)
//   p = exp(C - m), O += p V                                                                          (mma.sync)
// The GPU runs this at its power limit (B=32, H=32, Nk=32768, d=128: 990 W, 1.69 GHz), where every instruction costs
// bandwidth: with the conv as one load pair per FMA and P V as FMAs on widened values (~1000 instructions per 32 keys) the
// kernel sustained 5.56 TB/s; a plain read sustains 7.2.
// Both products take K and V as the 16-row A operand, as they lie in global memory.  K: rows are keys and the contraction
// index is permuted, so that a lane's fragment is contiguous pieces of a K row (Q, the 8-column B operand, is laid
// out to match once, in registers).  V: rows are head dims; a lane holds 16 or 32 bytes of 4 keys per MMA step, and a
// fragment register is two halfwords of neighbouring keys (one PRMT).  p stays fp32: columns 0, 1, 2 of the B operand are its
// bf16 parts hi, mid, lo (24 bits), whose products with V are exact; the three accumulator columns are added at the end.
// Warps are merged in shared memory, sub-splits (and, for small problems, the splits) inside a thread-block cluster, splits
// otherwise by combine_splits_kernel (result normalised into split 0, as the reference leaves it).  With `offset_causal` the
// score of a key later than a query row's own position is zeroed before the conv, as in the training forward, so that the
// result equals the last row of the training forward over the same sequence.
#pragma once
#include <cooperative_groups.h>

#include "fmta_common.cuh"
#include "fmta_params.h"

namespace fmta {

constexpr int kDecWarps = 4;
constexpr int kDecRing = 64;         // keys kept per warp for the conv window
constexpr int kDecRow = 68;          // ring row stride in floats: even rows 8 banks apart (no conflicts, stores or window loads)
constexpr int kDecMaxPages = 2048;   // block-table entries of one sequence kept in shared memory (paged cache)

// 16 or 32 bytes per lane, read once.  The 32-byte form lets the four lanes that share a K row of an MMA fragment fetch a whole
// 128-byte line with one instruction (with 16 bytes they fetch half of it, and the L2 sees twice the requests).  It needs K
// and V on 32-byte boundaries (rows are 128 or 256 bytes, so the bases decide); the callers' contract is 16 bytes, and the
// launcher takes the instantiations with two 16-byte loads (A32 = false) for bases in between.
FMTA_DEVINL void ldg_nc_v4(uint32_t* v, const void* p) {
  asm volatile("ld.global.nc.L1::no_allocate.L2::256B.v4.b32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "l"(p));
}
FMTA_DEVINL void ldg_nc_v8(uint32_t* v, const void* p) {
  asm volatile("ld.global.nc.L1::no_allocate.L2::256B.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "l"(p));
}
template <int W, bool A32>
FMTA_DEVINL void ldg_nc(uint32_t* v, const void* p, bool ok) {   // W words, zeros when !ok
  if (ok) {
    if (W == 8 && A32) {
      ldg_nc_v8(v, p);
    } else {
      ldg_nc_v4(v, p);
      if (W == 8) ldg_nc_v4(v + 4, reinterpret_cast<const unsigned char*>(p) + 16);
    }
  } else {
#pragma unroll
    for (int i = 0; i < W; ++i) v[i] = 0u;
  }
}

// keys handled by one split, a multiple of 16 * kDecWarps
__host__ __device__ inline int decode_keys_per_split(int Nk, int k_splits) {
  const int per = (Nk + k_splits - 1) / k_splits;
  return ((per + 16 * kDecWarps - 1) / (16 * kDecWarps)) * (16 * kDecWarps);
}

// NR: query rows per lane in the conv (2t, 2t + 1 and, from 9 rows on, 8 + those): 2 or 4.  CKP: filter width the taps are padded
// to with zeros (9: pad_k <= 4, 11: pad_k = 5, 17: any).  A32: K and V start on 32-byte boundaries.
template <int D, int NR, int CKP, bool PAGED, bool A32>
__global__ void __launch_bounds__(kDecWarps * 32, D == 128 ? 3 : 4) decode_kernel(const DecodeParams p) {
  constexpr int KS = D / 16;               // k-steps of the QK MMA
  constexpr int KW = D >= 64 ? 8 : 4;      // words of a K row per lane and load: 4 lanes cover 128 bytes (64 at d = 32)
  constexpr int KL = D / 8 / KW;           // loads per K row and lane
  constexpr bool R16 = NR > 2;
  constexpr int PKP = (CKP - 1) / 2, WC = (CKP <= 9) ? 3 : 5, W0 = 4 * ((WC - 1) / 2);   // conv window: WC float4 from 4g - W0 on
  constexpr bool THREG = NR * CKP <= 24;   // the lane's filter rows fit registers
  constexpr int VW = D == 128 ? 8 : 4;     // words of a V row per lane: 8 lanes cover the row (half of them idle at d = 32)
  __shared__ __align__(16) float sRing[kDecWarps][R16 ? 16 : 8][kDecRow];
  __shared__ __align__(16) float sTheta[16][20];
  __shared__ __align__(16) bf16 sPs[kDecWarps][4][32];     // hi, mid, lo of the step's probabilities, and a zero row
  __shared__ float sMergeO[kDecWarps][D];
  __shared__ float sMergeML[kDecWarps][2];
  __shared__ float sPartO[D];              // the CTA's partial, read by the other CTAs of the cluster
  __shared__ float sPartML[2];
  __shared__ int sTable[PAGED ? kDecMaxPages : 1];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int nsub = p.n_sub;
  const int split = blockIdx.x / nsub, sub = blockIdx.x - split * nsub, h = blockIdx.y, b = blockIdx.z;
  const int cq = p.cq, ck = p.ck, pk = (ck - 1) / 2;
  const int rows = min(p.q_len, cq);          // query rows that the last output row sees
  for (int i = tid; i < 16 * 20; i += kDecWarps * 32) (&sTheta[0][0])[i] = 0.f;
  if (tid < kDecWarps * 32) reinterpret_cast<uint2*>(&sPs[0][0][0])[tid] = make_uint2(0u, 0u);
  pdl_wait();
  pdl_trigger();
  // a per-sequence length comes from device memory the caller may have left stale: clamp it to the range the
  // block table (and the shared-memory copy of its row) was sized for
  const int Nk = (PAGED && p.seq_lens) ? min(max(p.seq_lens[b], 1), p.Nk) : p.Nk;
  const size_t bh = (size_t)b * p.H + h;
  // A 16-key tile never straddles a page (pages hold a multiple of 16 keys), so the page lookup is done once per tile:
  // tile_base(kb) is the address of key kb (a multiple of 16, clamped to the cache).
  auto tile_base = [&](const bf16* base, int kb) -> const bf16* {
    if (PAGED) {
      const int k = min(max(kb, 0), (Nk - 1) & ~15);
      return base + (((size_t)sTable[k >> p.page_shift] * p.H + h) * p.page_size + (k & (p.page_size - 1))) * D;
    }
    return base + (bh * (size_t)Nk + max(kb, 0)) * D;
  };
  if (PAGED) {
    const int npg = (Nk + p.page_size - 1) >> p.page_shift;
    for (int i = tid; i < npg; i += kDecWarps * 32) sTable[i] = p.block_table[(size_t)b * p.max_pages + i];
  }
  const bf16* Qg = p.Q + (bh * p.q_len + (p.q_len - rows)) * (size_t)D;
  __syncthreads();
  // theta rows that see a real query row: tap a = cq - rows + r  <->  ring row r; centred in CKP columns
  for (int i = tid; i < rows * ck; i += kDecWarps * 32)
    sTheta[i / ck][i % ck + PKP - pk] = p.theta[((size_t)h * cq + (cq - rows) + i / ck) * ck + (i % ck)];

  // B fragments of Q (column = query row) in the permuted-k layout (rows >= `rows` are zero)
  uint32_t qa[R16 ? 2 : 1][2 * KS];                         // word w: as the words of a K row
#pragma unroll
  for (int n = 0; n < (R16 ? 2 : 1); ++n)
#pragma unroll
    for (int c = 0; c < KL; ++c)
#pragma unroll
      for (int i = 0; i < KW; ++i)
        qa[n][c * KW + i] = g + 8 * n < rows ? *reinterpret_cast<const uint32_t*>(Qg + (size_t)(g + 8 * n) * D + c * 8 * KW + t * 2 * KW + 2 * i) : 0u;
  __syncthreads();
  auto row_of = [&](int r) { return 2 * t + (r & 1) + 8 * (r >> 1); };   // the lane's conv rows
  float th[THREG ? NR : 1][THREG ? CKP : 1];
  if constexpr (THREG) {
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
      for (int i = 0; i < CKP; ++i) th[r][i] = sTheta[row_of(r)][i];
  }

  // ---- key range of this warp: 32-key blocks from k_lo (a multiple of 16) on ----
  const int kps = decode_keys_per_split(Nk, p.k_splits);   // (per sequence when lengths differ)
  const int kpc = ((kps + nsub - 1) / nsub + 63) / 64 * 64; // keys per CTA
  const int kpw = (kpc / kDecWarps + 31) / 32 * 32;
  const int c_lo = split * kps + sub * kpc, c_hi = min(min(c_lo + kpc, (split + 1) * kps), Nk);
  const int k_lo = c_lo + warp * kpw, k_hi = min(k_lo + kpw, c_hi);
  const int nblk = k_hi > k_lo ? (k_hi - k_lo + 31) / 32 : 0;

  float m_run = -INFINITY, l_lane = 0.f;                     // l_lane: this lane's share of the sum
  float o[VW][4];                                            // [dims 2w, 2w + 1 of the lane's 2 VW][..]
#pragma unroll
  for (int i = 0; i < VW * 4; ++i) (&o[0][0])[i] = 0.f;
  float* ring = &sRing[warp][0][0];
  bf16* ps = &sPs[warp][0][0];
  uint32_t kf[2][2 * KS], vf[4][VW];

  auto load_k = [&](int kb) {                                // the 16-key tile at kb
    const bf16* src = tile_base(p.K, kb) + g * D + t * 2 * KW;
    const int lim = Nk - kb;                                 // rows of the tile inside the cache
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const bool ok = kb >= 0 && 8 * j + g < lim;
#pragma unroll
      for (int c = 0; c < KL; ++c) ldg_nc<KW, A32>(&kf[j][c * KW], src + 8 * j * D + c * 8 * KW, ok);
    }
  };
  auto load_v = [&](int kb, int sb) {                        // keys kb + 8 t + 4 sb + {0..3}: half of the 32-key block at kb
    const int k0 = kb + 8 * t + 4 * sb;
    const bf16* src = tile_base(p.V, kb + 16 * (t >> 1)) + (8 * (t & 1) + 4 * sb) * D + g * 2 * VW;
#pragma unroll
    for (int e = 0; e < 4; ++e) ldg_nc<VW, A32>(vf[e], src + e * D, k0 + e < Nk && (D >= 64 || g < 4));
  };
  auto scores = [&](int kb) {                                // S of the staged K tile -> ring
#pragma unroll
    for (int n = 0; n < (R16 ? 2 : 1); ++n) {                // query rows 8n ..
      float acc[4] = {0.f, 0.f, 0.f, 0.f};                   // (key g, rows 2t, 2t + 1), (key g + 8, the same)
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        const uint32_t a[4] = {kf[0][2 * s], kf[1][2 * s], kf[0][2 * s + 1], kf[1][2 * s + 1]};
        mma_bf16(acc, a, qa[n][2 * s], qa[n][2 * s + 1]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] *= p.scale;
      const int r0 = 8 * n + 2 * t;
      if (p.offset_causal && kb + 16 > Nk - rows) {          // only the last keys of the cache can lie in a row's future
        const int lim = Nk - rows + r0 - (kb + g);           // key offset from g of row r0's last key
        if (0 > lim) acc[0] = 0.f;
        if (0 > lim + 1) acc[1] = 0.f;
        if (8 > lim) acc[2] = 0.f;
        if (8 > lim + 1) acc[3] = 0.f;
      }
      const int col = (kb - k_lo + g) & (kDecRing - 1);      // col + 8 stays in the 16-key tile
      float* dst = ring + r0 * kDecRow + col;
      dst[0] = acc[0]; dst[kDecRow] = acc[1]; dst[8] = acc[2]; dst[kDecRow + 8] = acc[3];
    }
  };
  auto pv = [&](int sb) {                                    // O += p V for the staged half of the block
    const uint4 pa = *reinterpret_cast<const uint4*>(ps + min(g, 3) * 32 + 8 * t);
    const uint32_t b0 = sb ? pa.z : pa.x, b1 = sb ? pa.w : pa.y;
#pragma unroll
    for (int w = 0; w < VW; ++w) {
      const uint32_t a[4] = {__byte_perm(vf[0][w], vf[1][w], 0x5410), __byte_perm(vf[0][w], vf[1][w], 0x7632),
                             __byte_perm(vf[2][w], vf[3][w], 0x5410), __byte_perm(vf[2][w], vf[3][w], 0x7632)};
      mma_bf16(o[w], a, b0, b1);
    }
  };

  if (nblk > 0) {
    load_k(k_lo - 16);
    scores(k_lo - 16);
    load_k(k_lo);
    scores(k_lo);
    load_k(k_lo + 16);
#pragma unroll 1
    for (int i = 0; i < nblk; ++i) {
      // in flight here: the K tile at kb + 16 and the second V half of block i - 1
      const int kb = k_lo + 32 * i;
      scores(kb + 16);
      load_k(kb + 32);
      if (i > 0) pv(1);
      load_v(kb, 0);
      scores(kb + 32);
      if (i + 1 < nblk) load_k(kb + 48);
      __syncwarp();
      // ---- conv of block i: lane = keys 4g .. 4g+3 and its rows; then lane = key ----
      float c4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const float* row = ring + row_of(r) * kDecRow;
        float wv[4 * WC];
#pragma unroll
        for (int c = 0; c < WC; ++c) {
          const float4 x = *reinterpret_cast<const float4*>(row + 4 * ((8 * i + g - W0 / 4 + c) & (kDecRing / 4 - 1)));
          wv[4 * c] = x.x; wv[4 * c + 1] = x.y; wv[4 * c + 2] = x.z; wv[4 * c + 3] = x.w;
        }
#pragma unroll
        for (int bb = 0; bb < CKP; ++bb) {
          const float w = THREG ? th[THREG ? r : 0][THREG ? bb : 0] : sTheta[row_of(r)][bb];
#pragma unroll
          for (int e = 0; e < 4; ++e) c4[e] = fmaf(w, wv[bb + e + W0 - PKP], c4[e]);
        }
      }
      float cval;
      {
        const bool hi2 = t & 2, hi1 = t & 1;
        const float k0 = (hi2 ? c4[2] : c4[0]) + __shfl_xor_sync(0xffffffffu, hi2 ? c4[0] : c4[2], 2);
        const float k1 = (hi2 ? c4[3] : c4[1]) + __shfl_xor_sync(0xffffffffu, hi2 ? c4[1] : c4[3], 2);
        cval = (hi1 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, hi1 ? k0 : k1, 1);
      }
      if (kb + lane >= k_hi) cval = -INFINITY;
      float mx;
      asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(mx) : "f"(cval));
      if (mx > m_run) {                                      // warp-uniform
        const float alpha = exp2f((m_run - mx) * kLog2e);    // m_run = -inf -> 0
        m_run = mx;
        l_lane *= alpha;
#pragma unroll
        for (int q = 0; q < VW * 4; ++q) (&o[0][0])[q] *= alpha;
      }
      const float pj = exp2f((cval - m_run) * kLog2e);
      l_lane += pj;
      const bf16 p_hi = __float2bfloat16_rn(pj);
      const float r1 = pj - __bfloat162float(p_hi);
      const bf16 p_mid = __float2bfloat16_rn(r1);
      ps[lane] = p_hi; ps[32 + lane] = p_mid; ps[64 + lane] = __float2bfloat16_rn(r1 - __bfloat162float(p_mid));
      __syncwarp();
      pv(0);
      load_v(kb, 1);
    }
    pv(1);
  }
  // ---- columns hi + mid (lanes t = 0) + lo (t = 1), then the warps of the CTA ----
#pragma unroll
  for (int w = 0; w < VW; ++w)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float v = o[w][2 * u] + o[w][2 * u + 1];
      v += __shfl_down_sync(0xffffffffu, v, 1);
      if (v != v) v = o[w][2 * u];                           // an infinite V times a zero or negative rest of p: hi alone has its sign
      if (t == 0 && (D >= 64 || g < 4)) sMergeO[warp][g * 2 * VW + 2 * w + u] = v;
    }
  {
    const float l = warp_sum(l_lane);
    if (lane == 0) { sMergeML[warp][0] = m_run; sMergeML[warp][1] = l; }
  }
  __syncthreads();
  float m = -INFINITY;
#pragma unroll
  for (int w = 0; w < kDecWarps; ++w) m = fmaxf(m, sMergeML[w][0]);
  float wgt[kDecWarps], l = 0.f;
#pragma unroll
  for (int w = 0; w < kDecWarps; ++w) {
    wgt[w] = (sMergeML[w][0] == -INFINITY) ? 0.f : exp2f((sMergeML[w][0] - m) * kLog2e);
    l += sMergeML[w][1] * wgt[w];
  }
  float acc = 0.f;                                           // D <= 128 = blockDim.x: one head dim per thread
  if (tid < D)
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) acc += sMergeO[w][tid] * wgt[w];
  const size_t so = bh * p.k_splits + split;
  if (nsub == 1 && !p.fused) {
    if (tid < D) p.O_splits[so * D + tid] = acc;             // un-normalised partial
    if (tid == 0) { p.M_splits[so] = m; p.L_splits[so] = l; }
    return;
  }
  // ---- the CTAs of a split, and with `fused` all splits of the (batch, head), merge through distributed shared memory ----
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  if (tid < D) sPartO[tid] = acc;
  if (tid == 0) { sPartML[0] = m; sPartML[1] = l; }
  cl.sync();
  if (sub == 0) {
    const bool total = p.fused && split == 0;                // the merged, normalised result goes to split 0
    const int r0 = p.fused ? split * nsub : 0, r1 = total ? (int)cl.num_blocks() : r0 + nsub;
    float mm = -INFINITY, ll = 0.f, aa = 0.f;
    for (int r = r0; r < r1; ++r) mm = fmaxf(mm, cl.map_shared_rank(sPartML, r)[0]);
    for (int r = r0; r < r1; ++r) {
      const float* ml = cl.map_shared_rank(sPartML, r);
      const float w = (ml[0] == -INFINITY) ? 0.f : exp2f((ml[0] - mm) * kLog2e);
      ll += ml[1] * w;
      if (tid < D) aa += cl.map_shared_rank(sPartO, r)[tid] * w;
    }
    if (tid < D) p.O_splits[so * D + tid] = total ? aa / ll : aa;
    if (tid == 0) { p.M_splits[so] = mm; p.L_splits[so] = ll; }
  }
  cl.sync();                                                 // remote reads are done before a CTA's shared memory goes
}

// Merge the split partials of one (batch, head) and leave the normalised result in split 0
// (fwd_inference.cu:332-367 keeps the same convention).  The weights of the splits are made once, a thread each.
__global__ void __launch_bounds__(128) combine_splits_kernel(float* __restrict__ O_splits, float* __restrict__ M_splits,
                                                             float* __restrict__ L_splits, int k_splits, int D) {
  __shared__ float sW[128];
  __shared__ float sRed[4];
  const size_t bh = blockIdx.x;
  float* Ms = M_splits + bh * k_splits;
  float* Ls = L_splits + bh * k_splits;
  const int tid = threadIdx.x;
  pdl_wait();
  float m = -INFINITY;
  for (int s = tid; s < k_splits; s += 128) m = fmaxf(m, Ms[s]);
  m = warp_max(m);
  if ((tid & 31) == 0) sRed[tid >> 5] = m;
  __syncthreads();
  m = fmaxf(fmaxf(sRed[0], sRed[1]), fmaxf(sRed[2], sRed[3]));
  float l = 0.f, acc = 0.f;
  for (int s0 = 0; s0 < k_splits; s0 += 128) {
    const int n = min(128, k_splits - s0);
    __syncthreads();
    if (tid < n) {
      const float ms = Ms[s0 + tid], w = (ms == -INFINITY) ? 0.f : exp2f((ms - m) * kLog2e);
      sW[tid] = w;
      l += Ls[s0 + tid] * w;
    }
    __syncthreads();
    const float* src = O_splits + (bh * k_splits + s0) * D + tid;
    if (tid < D)
#pragma unroll 8
      for (int s = 0; s < n; ++s) acc += src[(size_t)s * D] * sW[s];
  }
  l = warp_sum(l);
  __syncthreads();
  if ((tid & 31) == 0) sRed[tid >> 5] = l;
  __syncthreads();
  l = (sRed[0] + sRed[1]) + (sRed[2] + sRed[3]);
  if (tid < D) O_splits[(bh * k_splits) * D + tid] = acc / l;
  if (tid == 0) { Ms[0] = m; Ls[0] = l; }
}

// Append n_new key/value rows per sequence to a paged cache: row r of sequence b goes to position
// seq_lens[b] + r (seq_lens is not modified; the caller advances it).  One 16-byte chunk per thread.
template <int D>
__global__ void kv_append_paged_kernel(bf16* __restrict__ Kpool, bf16* __restrict__ Vpool,
                                       const int* __restrict__ block_table, const int* __restrict__ seq_lens,
                                       const bf16* __restrict__ Knew, const bf16* __restrict__ Vnew, int H, int n_new,
                                       int page_size, int page_shift, int max_pages) {
  constexpr int CPR = D / 8;
  const int b = blockIdx.z;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;     // (head, row, chunk)
  pdl_wait();
  pdl_trigger();
  if (idx >= H * n_new * CPR) return;
  const int c = idx % CPR, r = (idx / CPR) % n_new, h = idx / (CPR * n_new);
  const int pos = seq_lens[b] + r;
  if (pos < 0 || (pos >> page_shift) >= max_pages) return;   // past the block table: the row is dropped, nothing is written
  const int pg = block_table[(size_t)b * max_pages + (pos >> page_shift)], in = pos & (page_size - 1);
  const size_t dst = (((size_t)pg * H + h) * page_size + in) * D + c * 8;
  const size_t src = (((size_t)b * H + h) * n_new + r) * D + c * 8;
  *reinterpret_cast<uint4*>(Kpool + dst) = *reinterpret_cast<const uint4*>(Knew + src);
  *reinterpret_cast<uint4*>(Vpool + dst) = *reinterpret_cast<const uint4*>(Vnew + src);
}

}  // namespace fmta

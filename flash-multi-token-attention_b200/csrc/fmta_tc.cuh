// Blackwell (sm_100a) primitives used by the stacked-GEMM forward kernel: mbarrier with bounded
// waits, TMA tensor loads (no multicast), tcgen05 MMA / commit / TMEM alloc / ld / st, and the
// shared-memory and instruction descriptors of tcgen05.mma.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "fmta_common.cuh"

namespace fmta {
namespace tc {

// ---------------------------------------------------------------- mbarrier
FMTA_DEVINL void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
FMTA_DEVINL void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
FMTA_DEVINL void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
FMTA_DEVINL void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
FMTA_DEVINL bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after kSpinLimit polls (or as soon as another thread has raised the
// CTA's abort flag) and returns false; the caller then leaves its loop and the kernel tears
// down normally.  No trap, no endless spin.
constexpr uint32_t kSpinLimit = 1u << 22;
FMTA_DEVINL bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint32_t limit = kSpinLimit) {
  for (uint32_t i = 0; i < limit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 1023u) == 1023u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}
// Poll limit of the wait that the expiry self-test makes run out: it waits on a barrier nothing
// ever arrives at, so a few hundred polls are enough to prove the point.
constexpr uint32_t kSelfTestSpinLimit = 256;

// ---------------------------------------------------------------- fences
FMTA_DEVINL void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
FMTA_DEVINL void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
FMTA_DEVINL void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---------------------------------------------------------------- TMA (tiled tensor loads)
// The innermost coordinate c0 times the element size is always a multiple of 16 bytes here
// (c0 is 0 or 64 bf16 elements); the other coordinates may be negative / out of range and
// then read zeros.
FMTA_DEVINL void tma_load_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// Tile store shared -> global (bulk async-group).  c0 = 0 and c1 >= 0 at every call: a store must not
// start at a negative coordinate; rows past the tensor's extent are clipped.
FMTA_DEVINL void tma_store_3d(const CUtensorMap* map, const void* smem_src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(map), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
// Contiguous copy shared -> global (bulk async-group; both addresses and the size multiples of 16 bytes) with an L2
// eviction-priority hint: data that is written once and read much later should not push the
// operands that are being re-read out of the cache.
FMTA_DEVINL uint64_t l2_policy_evict_first() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
FMTA_DEVINL void bulk_store_hint(void* gdst, const void* smem_src, uint32_t bytes, uint64_t policy) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group.L2::cache_hint [%0], [%1], %2, %3;"
               ::"l"(gdst), "r"(smem_u32(smem_src)), "r"(bytes), "l"(policy)
               : "memory");
}
// wait until every committed bulk store of this thread has completed (not only read its source)
FMTA_DEVINL void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
FMTA_DEVINL void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// wait until the committed stores have read their shared-memory source
FMTA_DEVINL void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
FMTA_DEVINL void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ---------------------------------------------------------------- TMEM
FMTA_DEVINL void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {   // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
}
FMTA_DEVINL void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
FMTA_DEVINL void tmem_dealloc(uint32_t taddr, uint32_t ncols) {     // whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 32 lanes x 32 columns of fp32: thread t of the warp gets lane (quarter base + t), 32 columns.
FMTA_DEVINL void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,"
      "%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
// 32 lanes x 16 columns.
FMTA_DEVINL void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
        "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
FMTA_DEVINL void tmem_ldn(uint32_t taddr, float (&v)[32]) { tmem_ld32(taddr, v); }
FMTA_DEVINL void tmem_ldn(uint32_t taddr, float (&v)[16]) { tmem_ld16(taddr, v); }
// Same without the trailing wait, for issuing several loads back to back (follow with tmem_wait_ld).
FMTA_DEVINL void tmem_ld32_nowait(uint32_t taddr, float (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,"
      "%28,%29,%30,%31}, [%32];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
        "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]),
        "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]),
        "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
      : "r"(taddr)
      : "memory");
}
FMTA_DEVINL void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
FMTA_DEVINL void tmem_st32(uint32_t taddr, const float (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31,%32};"
      ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
      "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
      "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])), "r"(__float_as_uint(v[8])),
      "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
      "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])),
      "r"(__float_as_uint(v[15])), "r"(__float_as_uint(v[16])), "r"(__float_as_uint(v[17])),
      "r"(__float_as_uint(v[18])), "r"(__float_as_uint(v[19])), "r"(__float_as_uint(v[20])),
      "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])), "r"(__float_as_uint(v[23])),
      "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])), "r"(__float_as_uint(v[26])),
      "r"(__float_as_uint(v[27])), "r"(__float_as_uint(v[28])), "r"(__float_as_uint(v[29])),
      "r"(__float_as_uint(v[30])), "r"(__float_as_uint(v[31]))
      : "memory");
}
FMTA_DEVINL void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------- tcgen05.mma
FMTA_DEVINL void tmem_st32u(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31,%32};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
      "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
      "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
      "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
// Named barrier among `count` threads (ids 1..15; 0 is __syncthreads).
FMTA_DEVINL void named_bar_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// ---- warp-uniform issue ------------------------------------------------------------------
// An MMA issuer warp runs its loop with all 32 lanes (so that descriptor arithmetic stays in
// uniform registers) and lets one elected lane execute each tcgen05 instruction; the elected
// lane is the same for a given member mask, so commits track the MMAs issued before them.
FMTA_DEVINL bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
  return pred != 0;
}
FMTA_DEVINL bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}
// D[tmem] (+)= A * B, kind::f16 (bf16 inputs, fp32 accumulate).  Descriptors come as (constant high word, low word): the low
// word holds the start address, so stepping through an operand is a 32-bit add.  ss: both operands in shared memory; ts: A in
// tensor memory (128 lanes = rows, each 32-bit column = 2 consecutive K elements).
// Elections and MMAs sit in one asm block, the MMAs PREDICATED on the elected lane.  Behind a branch (`if (elect_one())`
// around each MMA) every operand goes through the reconvergence of the warp and back into uniform registers: back to back
// that took 101-108 cycles per MMA whatever its size; predicated, 39 cycles at N = 16 and the tensor core's own rate above
// (64 cycles for 128 x 128 x 16, 43 for a pair's 256 x 64 x 16).
template <int ACC>
FMTA_DEVINL void mma_ss2e(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "n"(ACC)
      : "memory");
}
FMTA_DEVINL void mma_ss2pe(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
FMTA_DEVINL void mma_commit_e(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar))
      : "memory");
}
// Four MMAs of one chain: operands as_ and bs_ (descriptor units of 16 bytes; tensor-memory columns for a TMEM A) apart,
// the first one overwriting unless `accumulate`.  G = 2: of a CTA pair.
#define FMTA_MMA4_SS(CG)                                                                                          \
  asm volatile(                                                                                                  \
      "{\n\t.reg .pred p, q, t;\n\t.reg .b64 da, db;\n\t"                                                           \
      "elect.sync _|q, 0xffffffff;\n\t"                                                                           \
      "setp.ne.b32 p, %12, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"                                                           \
      "mov.b64 da, {%1, %9};\n\tmov.b64 db, {%5, %10};\n\t"                                                          \
      "@q tcgen05.mma.cta_group::" CG ".kind::f16 [%0], da, db, %11, p;\n\t"                                        \
      "mov.b64 da, {%2, %9};\n\tmov.b64 db, {%6, %10};\n\t"                                                          \
      "@q tcgen05.mma.cta_group::" CG ".kind::f16 [%0], da, db, %11, t;\n\t"                                        \
      "mov.b64 da, {%3, %9};\n\tmov.b64 db, {%7, %10};\n\t"                                                          \
      "@q tcgen05.mma.cta_group::" CG ".kind::f16 [%0], da, db, %11, t;\n\t"                                        \
      "mov.b64 da, {%4, %9};\n\tmov.b64 db, {%8, %10};\n\t"                                                          \
      "@q tcgen05.mma.cta_group::" CG ".kind::f16 [%0], da, db, %11, t;\n\t}"                                       \
      ::"r"(d_tmem), "r"(a_lo), "r"(a_lo + as_), "r"(a_lo + 2 * as_), "r"(a_lo + 3 * as_), "r"(b_lo), "r"(b_lo + bs_), \
      "r"(b_lo + 2 * bs_), "r"(b_lo + 3 * bs_), "r"(a_hi), "r"(b_hi), "r"(idesc), "r"(accumulate)                   \
      : "memory")
#define FMTA_MMA4_TS(CG)                                                                                          \
  asm volatile(                                                                                                  \
      "{\n\t.reg .pred p, q, t;\n\t.reg .b64 db;\n\t"                                                               \
      "elect.sync _|q, 0xffffffff;\n\t"                                                                           \
      "setp.ne.b32 p, %11, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"                                                           \
      "mov.b64 db, {%5, %9};\n\t@q tcgen05.mma.cta_group::" CG ".kind::f16 [%0], [%1], db, %10, p;\n\t"             \
      "mov.b64 db, {%6, %9};\n\t@q tcgen05.mma.cta_group::" CG ".kind::f16 [%0], [%2], db, %10, t;\n\t"             \
      "mov.b64 db, {%7, %9};\n\t@q tcgen05.mma.cta_group::" CG ".kind::f16 [%0], [%3], db, %10, t;\n\t"             \
      "mov.b64 db, {%8, %9};\n\t@q tcgen05.mma.cta_group::" CG ".kind::f16 [%0], [%4], db, %10, t;\n\t}"            \
      ::"r"(d_tmem), "r"(a_tmem), "r"(a_tmem + as_), "r"(a_tmem + 2 * as_), "r"(a_tmem + 3 * as_), "r"(b_lo),       \
      "r"(b_lo + bs_), "r"(b_lo + 2 * bs_), "r"(b_lo + 3 * bs_), "r"(b_hi), "r"(idesc), "r"(accumulate)             \
      : "memory")
template <int G = 1>
FMTA_DEVINL void mma4_ss(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t as_, uint32_t b_lo, uint32_t b_hi, uint32_t bs_,
                         uint32_t idesc, uint32_t accumulate) {
  if constexpr (G == 1) FMTA_MMA4_SS("1"); else FMTA_MMA4_SS("2");
}
template <int G = 1>
FMTA_DEVINL void mma4_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t as_, uint32_t b_lo, uint32_t b_hi, uint32_t bs_, uint32_t idesc,
                         uint32_t accumulate) {
  if constexpr (G == 1) FMTA_MMA4_TS("1"); else FMTA_MMA4_TS("2");
}
#undef FMTA_MMA4_SS
#undef FMTA_MMA4_TS

// ---- CTA pairs (cta_group::2) --------------------------------------------------------------
// The two CTAs of a cluster of 2 work on one 256-row MMA: each holds its 128 rows of A and of the accumulator and
// HALF of the B tile; the CTA of rank 0 issues for both.  Shared-memory operands sit at the same offsets in both CTAs,
// barriers the issuer waits on live in rank 0's shared memory, commits arrive in both.
FMTA_DEVINL uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
FMTA_DEVINL uint32_t cluster_addr(const void* smem, uint32_t rank) {      // shared::cluster address of the same variable in CTA `rank`
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(smem)), "r"(rank));
  return a;
}
FMTA_DEVINL void cluster_sync_all() {     // every thread of both CTAs
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
FMTA_DEVINL void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
FMTA_DEVINL void st_cluster_u32(uint32_t cluster_dst, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_dst), "r"(v) : "memory");
}
// One look at a barrier, no waiting.
FMTA_DEVINL uint32_t mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok;
}
// The issuer's end of a ring of tiles.  The tensor core takes an MMA only when the one before it is under way, so whatever
// the issuer does between two tiles leaves it idle: a wait that is over already still costs 200 cycles.  take() therefore
// looks at the NEXT tile's barrier before the MMAs of this one are issued and give() picks the answer up behind them.
// G = 2: of a CTA pair (the slots are released in both CTAs).
template <int NSLOT, int G = 2>
struct TileRing {
  uint64_t *full, *empty;
  volatile int* abort_flag;
  int slot = 0, ph = 0, nslot = 0, nph = 0;
  uint32_t seen = 0;
  bool ready = false;
  FMTA_DEVINL TileRing(uint64_t* f, uint64_t* e, volatile int* a) : full(f), empty(e), abort_flag(a) {}
  FMTA_DEVINL bool take() {
    if (!ready && !mbar_wait_warp(&full[slot], ph, abort_flag)) return false;
    tc_fence_after();
    nslot = slot + 1 == NSLOT ? 0 : slot + 1;
    nph = nslot == 0 ? ph ^ 1 : ph;
    seen = mbar_test(&full[nslot], nph);
    return true;
  }
  FMTA_DEVINL void give();
};
// tile into this CTA's shared memory, completing on a barrier of rank 0 (cluster_bar: shared::cluster address)
FMTA_DEVINL void tma_load_3d_pair(void* smem_dst, const CUtensorMap* map, uint32_t cluster_bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(cluster_bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
FMTA_DEVINL void tmem_alloc_pair(uint32_t* smem_dst, uint32_t ncols) {    // one warp of each CTA
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
FMTA_DEVINL void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {      // one warp of each CTA
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// arrive on the barrier at this offset in both CTAs once all MMAs issued so far by this thread have completed
FMTA_DEVINL void mma_commit_pair(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
      ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

template <int NSLOT, int G>
FMTA_DEVINL void TileRing<NSLOT, G>::give() {
  if constexpr (G == 2) mma_commit_pair(&empty[slot]); else mma_commit_e(&empty[slot]);
  slot = nslot; ph = nph;
  ready = __all_sync(0xffffffffu, seen);
}

// CTAs are dispatched in linear block order.  The row blocks of a (batch, head) pair run side by side, longest first, and
// share its K-tilde and V in L2; the last `X` pairs (a few waves of the GPU) are walked length-major, so that the greedy
// hardware scheduler ends with the short CTAs.
FMTA_DEVINL void pair_block_order(int lin, int nqb, int nBH, int& bh, int& r) {
  const int X = min(nBH, max(1, (256 + nqb / 2) / nqb));
  const int head = (nBH - X) * nqb;
  if (lin < head) { bh = lin / nqb; r = lin - bh * nqb; }
  else { lin -= head; r = lin / X; bh = nBH - X + (lin - r * X); }
}

// Instruction descriptor, kind::f16: bf16 x bf16 -> fp32, M x N tile.
//   bits [4,6) D format (1 = F32); [7,10) A format (1 = BF16); [10,13) B format (1 = BF16);
//   bit 15 A major (0 = K, 1 = MN); bit 16 B major; [17,23) N >> 3; [24,29) M >> 4.
__host__ __device__ constexpr uint32_t make_idesc(int M, int N, int a_mn_major, int b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn_major << 15) | ((uint32_t)b_mn_major << 16) |
         ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Shared-memory matrix descriptor.
//   bits [0,14) start address >> 4; [16,30) leading byte offset >> 4; [32,46) stride byte offset >> 4;
//   [46,48) version = 1; [61,64) layout: 0 = no swizzle ("interleaved" 8x16-byte core matrices),
//   2 = 128-byte swizzle, 4 = 64-byte swizzle.
constexpr uint64_t kLayoutNone = 0, kLayoutSW128 = 2, kLayoutSW64 = 4;
FMTA_DEVINL uint64_t make_sdesc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint64_t layout) {
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (layout << 61);
}

}  // namespace tc
}  // namespace fmta

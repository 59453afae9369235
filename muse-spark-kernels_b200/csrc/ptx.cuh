// Thin inline-PTX wrappers for sm_100a: mbarrier, bulk async copies (TMA engine),
// cp.async, tcgen05 (TMEM allocation, MMA, commit, ld/st) and the FP4/FP8 converts.
//
// Rules this file keeps:
//  * no cluster-multicast load of any kind is defined here;
//  * every wait is bounded: a poll loop gives up after MSK_WAIT_LIMIT_NS of wall
//    time (or at once when the CTA's abort word is set), the caller records an
//    error code and unwinds; nothing traps and nothing spins for ever.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace msk {

#ifndef MSK_WAIT_LIMIT_NS
#define MSK_WAIT_LIMIT_NS 1000000000ull  // one second
#endif

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t) : : "memory");  // the clobber pins it between barriers
  return t;
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
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

// try_wait that lets the hardware park the thread for up to `hint_ns` while the phase is
// incomplete (it resumes as soon as the phase completes). Without the hint the poll loop of
// a waiting warp spins fast enough to take issue slots from the working warps of its
// scheduler: measured here, five spinning warps slowed the MMA-issuing warp about sixfold.
__device__ __forceinline__ bool mbar_try_wait_parked(uint64_t* bar, uint32_t parity, uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}

// Bounded wait on an mbarrier phase. `abort_word` is a CTA-shared int that any
// role sets non-zero when it gave up; a set word makes every later wait return
// false at once so that all roles unwind together. Returns true when the phase
// completed.
// The polling part is one shared function, not inlined at the several dozen call sites: a step of one
// token starts with a cold instruction cache, and every copy of this loop that a role runs into for the
// first time would be another line to fetch from memory.
__device__ __noinline__ bool mbar_wait_poll(uint32_t bar_addr, uint32_t parity, volatile int* abort_word) {
  const uint64_t t0 = globaltimer_ns();
  uint32_t polls = 0;
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar_addr), "r"(parity), "r"(4000u)
        : "memory");
    if (ok) return true;
    if ((++polls & 15u) == 0u) {
      if (*abort_word != 0) return false;
      if (globaltimer_ns() - t0 > MSK_WAIT_LIMIT_NS) {
        *abort_word = 1;
        return false;
      }
    }
  }
}

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_word) {
  if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait_poll(smem_u32(bar), parity, abort_word);
}

// The same wait with the polling loop inlined: for the wide token tiles, whose warps wait at every
// stage of a long, warm main loop (measured: the call cost the 8192-token step about 10 %).
__device__ __forceinline__ bool mbar_wait_inline(uint64_t* bar, uint32_t parity, volatile int* abort_word) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t polls = 0;
  while (true) {
    if (mbar_try_wait_parked(bar, parity, 4000u)) return true;
    if ((++polls & 15u) == 0u) {
      if (*abort_word != 0) return false;
      if (globaltimer_ns() - t0 > MSK_WAIT_LIMIT_NS) {
        *abort_word = 1;
        return false;
      }
    }
  }
}

// The same wait, acquiring what threads of the other CTAs of the cluster have released by their arrives.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_word) {
  const uint64_t t0 = globaltimer_ns();
  uint32_t polls = 0;
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(4000u)
        : "memory");
    if (ok) return true;
    if ((++polls & 15u) == 0u) {
      if (*abort_word != 0) return false;
      if (globaltimer_ns() - t0 > MSK_WAIT_LIMIT_NS) {
        *abort_word = 1;
        return false;
      }
    }
  }
}

// The same wait for a whole warp, with one outcome: every lane polls for itself (and so acquires what the barrier publishes),
// and the warp goes on once all lanes have seen the phase complete, or gives up together. Lanes that gave up one by one
// would leave the others behind in full-warp instructions. All 32 lanes call it.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_word) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t polls = 0;
  while (true) {
    if (__all_sync(0xffffffffu, mbar_try_wait_parked(bar, parity, 4000u))) return true;
    if ((++polls & 15u) == 0u && __any_sync(0xffffffffu, *abort_word != 0 || globaltimer_ns() - t0 > MSK_WAIT_LIMIT_NS)) {
      *abort_word = 1;
      return false;
    }
  }
}

// The same wait for hand-offs that complete within a few hundred cycles (the 128 epilogue threads
// meeting at their barrier): poll without parking first, so that the wake-up latency of a parked
// thread is not paid on every meeting; then fall back to the parked wait.
__device__ __forceinline__ bool mbar_wait_short(uint64_t* bar, uint32_t parity, volatile int* abort_word) {
#pragma unroll 1
  for (int i = 0; i < 64; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return mbar_wait(bar, parity, abort_word);
}

// Non-blocking probe of a phase (mbarrier.test_wait): true when the phase has completed. Unlike
// try_wait it never suspends the thread, so it tells whether a wait that follows will have to wait.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// ------------------------------------------------------- async-proxy fences
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Between generic and asynchronous accesses of any state space (rows another SM has stored, about to be read by
// a bulk copy).
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// Named barrier over `threads` threads of the CTA (all of them take part; no early exits in between).
__device__ __forceinline__ void named_bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Counters in global memory: release on the writer's side, acquire on the reader's.
__device__ __forceinline__ void red_release_add(unsigned int* p, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// The same between the warps of a CTA, in shared memory.
__device__ __forceinline__ int ld_acquire_cta(const int* p) {
  int v;
  asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_cta(int* p, int v) {
  asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}

// ----------------------------------------------------- bulk copy (TMA, 1-D)
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ uint64_t policy_evict_normal() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
// global -> this CTA's shared memory; both addresses 16-byte aligned, bytes % 16 == 0.
__device__ __forceinline__ void bulk_g2s(void* smem_dst, const void* gmem_src, uint32_t bytes, uint64_t* bar,
                                         uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
      ::"r"(smem_u32(smem_dst)), "l"(gmem_src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}
// 2-D tiled TMA load (no multicast): box of the tensor map at element coordinates (c0 inner,
// c1 outer) -> this CTA's shared memory, completing on `bar`. c0 * element size must be a
// multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const void* tmap, int c0, int c1, uint64_t* bar,
                                            uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3}], [%4], %5;" ::"r"(smem_u32(smem_dst)),
      "l"(tmap), "r"(c0), "r"(c1), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}
// The same from a tensor of three dimensions.
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const void* tmap, int c0, int c1, int c2, uint64_t* bar,
                                            uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(smem_u32(smem_dst)),
      "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}
// L2 prefetch of a contiguous piece (16-byte aligned, a multiple of 16 bytes).
__device__ __forceinline__ void bulk_prefetch_l2(const void* gmem, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void prefetch_tensormap(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}

// ------------------------------------------------------------ clusters
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 16 bytes at this CTA's shared address `addr`, as CTA `rank` of the cluster holds them.
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// This CTA's shared address `addr` as a cluster address of CTA `rank`.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  return a;
}
// 16 bytes into the shared memory of any CTA of the cluster, counted on a barrier of that CTA (both cluster addresses).
__device__ __forceinline__ void st_async_v4(uint32_t addr, int4 v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "r"(v.x),
               "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
               : "memory");
}
// Arrive on a barrier of any CTA of the cluster (a cluster address). The relaxed form is for what lies in TMEM, ordered by the
// tcgen05 fences; the other one releases this thread's reads and writes of memory as well, and so waits for all of its stores to
// global memory (in place of the relaxed one everywhere the pair kernel took a third longer).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_release_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx_cluster(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// 3-D tiled TMA load into this CTA's shared memory that completes on a barrier of either CTA of the pair (a cluster address).
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const void* tmap, int c0, int c1, int c2, uint32_t bar,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(smem_u32(smem_dst)),
      "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(bar), "l"(policy)
      : "memory");
}

// ------------------------------------------------------------ cp.async 16 B
__device__ __forceinline__ void cp_async16_hint(void* smem_dst, const void* gmem_src, bool valid, uint64_t policy) {
  // src-size 0 zero-fills the 16 destination bytes (used for padding rows).
  const uint32_t sz = valid ? 16u : 0u;
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;" ::"r"(smem_u32(smem_dst)),
               "l"(gmem_src), "r"(sz), "l"(policy)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ------------------------------------------------------------------ tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Arrive (count 1) on `bar` once every tcgen05.mma issued so far by this thread
// has completed. Implies tcgen05.fence::before_thread_sync.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// The same for a pair of CTAs (cta_group::2): allocation and release are made by one warp of either CTA, MMAs and commits by
// one thread of CTA 0; a commit arrives on the barrier at this offset in both CTAs.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   smem_u32(bar)),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}
// One MMA of a run over K: B lies `o` behind descriptor half `l` (units of 16 bytes; an address never carries out of the low half), A
// `c` columns behind the first. By a single thread (elect_one() around the whole loop of an issuer): measured beside sixteen
// decoding warps, an MMA of 32 columns issues every 16 cycles this way, every 50 to 70 where the warp elects a lane, issues and meets
// again for each run.
#define MSK_MMA_STEP(group, d, a, l, o, c, idesc, acc)                                                  \
  "add.u32 x, " l ", " o ";\n\tmov.b64 b, {x, hi};\n\tadd.u32 c, " a ", " c ";\n\t"                       \
  "tcgen05.mma.cta_group::" group ".kind::f16 [" d "], [c], b, " idesc ", " acc ";\n\t"

// D[256 rows over both CTAs' TMEM, N] (+)= A[256 rows, 256] (128 rows in either TMEM) * B[N, 256] (N / 2 rows in either CTA): the
// sixteen MMAs of a K stage (two slots) by one thread, and the commits that hand its slots back in both CTAs (empty_bar and
// the barrier behind it). The answer of a probe of `next_full` (true: complete) is asked for before the MMAs and read behind them, so
// that its latency hides behind the issue. b_desc: the first of four sub-tiles of 64 K, which lie `sub` apart (units of 16 bytes).
__device__ __forceinline__ bool mma_stage_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate,
                                               uint32_t empty_bar, uint32_t next_full, uint32_t parity, uint32_t sub) {
  uint32_t ok;
#define MSK_PAIR_COMMIT(bar) "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [" bar "], %10;\n\t"
#define MSK_PAIR_STEP(l, o, c, acc) MSK_MMA_STEP("2", "%1", "%2", l, o, c, "%4", acc)
  asm volatile(
      "{\n\t.reg .pred q, acc, t;\n\t.reg .b32 l0, l1, l2, l3, hi, second, x, c;\n\t.reg .b64 b;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%7], %8;\n\t"
      "setp.ne.b32 acc, %5, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "mov.b64 {l0, hi}, %3;\n\tadd.u32 l1, l0, %9;\n\tadd.u32 l2, l1, %9;\n\tadd.u32 l3, l2, %9;\n\tadd.u32 second, %6, 8;\n\t"
      MSK_PAIR_STEP("l0", "0", "0", "acc") MSK_PAIR_STEP("l0", "2", "8", "t")
      MSK_PAIR_STEP("l0", "4", "16", "t") MSK_PAIR_STEP("l0", "6", "24", "t")
      MSK_PAIR_STEP("l1", "0", "32", "t") MSK_PAIR_STEP("l1", "2", "40", "t")
      MSK_PAIR_STEP("l1", "4", "48", "t") MSK_PAIR_STEP("l1", "6", "56", "t")
      MSK_PAIR_COMMIT("%6")
      MSK_PAIR_STEP("l2", "0", "64", "t") MSK_PAIR_STEP("l2", "2", "72", "t")
      MSK_PAIR_STEP("l2", "4", "80", "t") MSK_PAIR_STEP("l2", "6", "88", "t")
      MSK_PAIR_STEP("l3", "0", "96", "t") MSK_PAIR_STEP("l3", "2", "104", "t")
      MSK_PAIR_STEP("l3", "4", "112", "t") MSK_PAIR_STEP("l3", "6", "120", "t")
      MSK_PAIR_COMMIT("second")
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(ok)
      : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(empty_bar), "r"(next_full), "r"(parity),
        "r"(sub), "h"(static_cast<uint16_t>(3))
      : "memory");
#undef MSK_PAIR_STEP
#undef MSK_PAIR_COMMIT
  return ok != 0;
}

// Shared-memory matrix descriptor, K-major, no swizzle ("interleave"): the tile is
// a grid of 8-row x 16-byte core matrices, each 128 contiguous bytes.
//   lbo = byte distance between core matrices adjacent in K,
//   sbo = byte distance between 8-row groups (M or N direction).
__device__ __forceinline__ uint64_t smem_desc_kmajor_noswz(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;  // descriptor version for sm_100
  return d;         // layout type 0 = no swizzle, base offset 0
}

// Shared-memory matrix descriptor, K-major, 128-byte swizzle: rows of 128 bytes (64 BF16),
// 8-row groups 1024 bytes apart, as written by a TMA load with CU_TENSOR_MAP_SWIZZLE_128B.
// The tile base must be 1024-byte aligned; a K step of 16 elements advances saddr by 32 bytes.
__device__ __forceinline__ uint64_t smem_desc_kmajor_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(1) << 16;          // leading byte offset: unused with swizzled K-major
  d |= static_cast<uint64_t>(1024 >> 4) << 32;  // stride byte offset between 8-row groups
  d |= 1ull << 46;                              // descriptor version for sm_100
  d |= 2ull << 61;                              // layout type: 128-byte swizzle
  return d;
}

// Instruction descriptor for kind::f16: D = FP32, A/B = F16 (0) or BF16 (1), both K-major.
enum : uint32_t { FMT_F16 = 0, FMT_BF16 = 1 };
__host__ __device__ constexpr uint32_t idesc_f16(uint32_t a_fmt, uint32_t b_fmt, uint32_t M, uint32_t N) {
  return (1u << 4) | (a_fmt << 7) | (b_fmt << 10) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]; A: lane = row, one 32-bit column = two consecutive K elements. The eight MMAs of an A slot (128 K) by
// one thread: B of K step j lies (j & 3) * STEP + (j >> 2) * sub behind b_desc (units of 16 bytes).
template <int STEP>
__device__ __forceinline__ void mma_slot_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate,
                                            uint32_t sub) {
#define MSK_SLOT_STEP(l, o, c, acc) MSK_MMA_STEP("1", "%0", "%1", l, o, c, "%3", acc)
  asm volatile(
      "{\n\t.reg .pred acc, t;\n\t.reg .b32 l0, l1, hi, x, c;\n\t.reg .b64 b;\n\t"
      "setp.ne.b32 acc, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "mov.b64 {l0, hi}, %2;\n\tadd.u32 l1, l0, %5;\n\t"
      MSK_SLOT_STEP("l0", "0", "0", "acc") MSK_SLOT_STEP("l0", "%6", "8", "t")
      MSK_SLOT_STEP("l0", "%7", "16", "t") MSK_SLOT_STEP("l0", "%8", "24", "t")
      MSK_SLOT_STEP("l1", "0", "32", "t") MSK_SLOT_STEP("l1", "%6", "40", "t")
      MSK_SLOT_STEP("l1", "%7", "48", "t") MSK_SLOT_STEP("l1", "%8", "56", "t")
      "}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(sub), "n"(STEP), "n"(2 * STEP), "n"(3 * STEP)
      : "memory");
#undef MSK_SLOT_STEP
}
#undef MSK_MMA_STEP

// 32 lanes x 32 bit, N consecutive columns per thread. The warp may only touch
// TMEM lanes [32*(warp_id%4), +32); the lane base goes in bits 31..16 of taddr.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// ---------------------------------------------------- register-operand MMA
// D[16 x 8] += A[16 x 16] * B[16 x 8], F16 operands, FP32 accumulators. Lane (r = lane / 4, q = lane % 4): a0
// row r, K 2q and 2q+1; a1 row r+8; a2, a3 the same at K + 8; b0, b1 column r at those K; d0, d1 row r, columns
// 2q and 2q+1; d2, d3 row r+8. Measured on B200: one per 8.3 cycles and scheduler.
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ------------------------------------------------------------ FP4/FP8 decode
// Four bytes = eight E2M1 codes (low nibble first) -> four f16x2 registers.
__device__ __forceinline__ void cvt_e2m1x8_f16(uint32_t w, uint32_t& h01, uint32_t& h23, uint32_t& h45,
                                               uint32_t& h67) {
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
      "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
      "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
      : "=r"(h01), "=r"(h23), "=r"(h45), "=r"(h67)
      : "r"(w));
}
// Two E4M3 bytes (low byte first) -> f16x2.
__device__ __forceinline__ uint32_t cvt_e4m3x2_f16(uint16_t two) {
  uint32_t h;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h) : "h"(two));
  return h;
}
__device__ __forceinline__ uint32_t hmul2_f16(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}

// ---------------------------------------------- programmatic dependent launch
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace msk

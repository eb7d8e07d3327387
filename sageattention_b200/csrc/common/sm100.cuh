// Thin inline-PTX layer for sm_100a: mbarrier, TMA (cp.async.bulk.tensor), tcgen05
// (TMEM allocation, block-scaled MMA, tcgen05.cp/ld/st, commit) and descriptor builders.
//
// Every wait in this file is BOUNDED: a wait that exceeds its budget records a status word and returns false instead of
// spinning forever.  A wait for data has 2^20 probes that suspend for up to 2 us each (about two seconds), or 2^24
// plain polls; once a CTA has recorded an error all of its later waits for data return after a failed
// probe (256 plain polls).  The hand-over of work items goes on after an error and has four times that budget
// (mbar_wait_item).  So a protocol bug ends a kernel within seconds, with a readable status, instead of hanging the device.
#pragma once
#include <cuda_runtime.h>
#include <cuda.h>
#include <stdint.h>

namespace nvfp4 {

// ---------------------------------------------------------------------------------------
// status codes written by kernels into their device status word (0 = ok)
// ---------------------------------------------------------------------------------------
enum : int {
  KSTAT_OK = 0,
  KSTAT_WAIT_TIMEOUT = 0x100,  // | site id
};

#ifndef NVFP4_WAIT_SPINS
#define NVFP4_WAIT_SPINS (1u << 20)
#endif

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Number of the warp in its block, as a broadcast: the compiler then knows that all lanes hold the same and keeps what
// follows from it in uniform registers -- tensor-memory addresses, of which tcgen05 takes no others, barriers, roles.
// From threadIdx.x / 32 alone it moves every such address over, one by one, and holds them in (spilled) registers.
// Whole passes, results the same to the bit: prefill Z4 S8192 1837 -> 1748 us, padded cross attention 95.0 -> 87.7, training
// steps of 16384 packed tokens 1660 -> 1578 and of S8192 D256 1530 -> 1485; decode, bound elsewhere, +-2 %.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "elect.sync _|P, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}\n"
      : "=r"(pred));
  return pred != 0;
}

// ------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// One potentially-blocking probe: the hardware may park the thread until the phase completes or
// the hint (ns) runs out, so a waiting warp costs few issue slots.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(2000u)
      : "memory");
  return ok != 0;
}

// Non-blocking probe (cheap when the phase has already completed).
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait with an explicit probe budget. `err` is a CTA-shared int (0 = healthy). Returns
// false on timeout, after recording KSTAT_WAIT_TIMEOUT | site in `err`.  Not unrolled: a kernel has some twenty
// waits, and unrolled by four they were half of its code (forward D = 128 86 -> 38 KB), which its warps fetch in
// different places at once.  Whole passes: prefill Z4 H32 Hk8 S8192 2183 -> 2134 us, cross attention Z2 H32 Sq1029
// Skv2309 127.5 -> 123.1, training step S8192 D256 1884 -> 1855.
__device__ __forceinline__ bool mbar_wait_n(uint64_t* bar, uint32_t parity, volatile int* err,
                                            int site, uint32_t spins) {
  if (mbar_test_wait(bar, parity)) return true;      // a completed phase costs less this way than by try_wait
#pragma unroll 1
  for (uint32_t i = 0; !mbar_try_wait(bar, parity); ++i) {
    if (*err) return false;
    if (i >= spins) {
      *err = KSTAT_WAIT_TIMEOUT | site;
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* err,
                                          int site) {
  return mbar_wait_n(bar, parity, err, site, NVFP4_WAIT_SPINS);
}

// Two barriers at once.  A probe takes 100 to 150 clocks even where the phase has long completed, and a warp that
// waits for one barrier after the other pays them one after the other; probed together their latencies overlap.
__device__ __forceinline__ void mbar_wait_all(uint64_t* a, uint32_t pa, uint64_t* b, uint32_t pb, volatile int* err, int site) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P, Q;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 Q, [%3], %4;\n\t"
      "and.pred P, P, Q;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(a)), "r"(pa), "r"(smem_u32(b)), "r"(pb)
      : "memory");
  if (ok) return;
  mbar_wait(a, pa, err, site);
  mbar_wait(b, pb, err, site);
}

// The same by a whole warp of which one thread then acts: commits products, loads, arrives.  No lane may be left behind in a
// wait, for what that thread does lets the barrier go on, and by its next phase the parity that a late lane looks for would
// be gone again.  Where several waits stand in front of one act, the lanes meet once, behind the last: after each of them
// the bf16 backward D128 S4096 took 107.6 us instead of 106.5, the forward S4096 not causal 213.1 instead of 212.8 (never
// meeting, 106.2 and 211.9).
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* err, int site) {
  const bool ok = mbar_wait(bar, parity, err, site);
  __syncwarp();
  return ok;
}

// Bounded wait that polls without parking the thread: lowest wake-up latency, meant for a lone
// elected thread (an MMA issuer) whose reaction time is on the critical path.
__device__ __forceinline__ bool mbar_spin_wait(uint64_t* bar, uint32_t parity, volatile int* err,
                                               int site) {
#pragma unroll 1
  for (uint32_t i = 0; !mbar_test_wait(bar, parity); ++i) {
    if ((i & 255u) == 255u && *err) return false;
    if (i >= (NVFP4_WAIT_SPINS << 4)) {
      *err = KSTAT_WAIT_TIMEOUT | site;
      return false;
    }
  }
  return true;
}

// Wait of a hand-over of work items, by a whole warp or by one thread.  It goes on when the CTA has recorded an error, so
// that all warps keep to the same sequence of items (and of the barriers in them) until the last one: by the time that
// the budget, four times that of a data wait, runs out, an expired data wait has let everything else drain.  False when
// it has run out: what was to be handed over is not there, and the caller leaves its loop over the items.
__device__ __forceinline__ bool mbar_wait_item_n(uint64_t* bar, uint32_t parity, volatile int* err, int site, uint32_t spins) {
#pragma unroll 1
  for (uint32_t i = 0; !mbar_try_wait(bar, parity); ++i)
    if (i >= spins) {
      if (*err == 0) *err = KSTAT_WAIT_TIMEOUT | site;      // the first expired wait is the one to look at
      return false;
    }
  return true;
}
__device__ __forceinline__ bool mbar_wait_item(uint64_t* bar, uint32_t parity, volatile int* err, int site) {
  return mbar_wait_item_n(bar, parity, err, site, NVFP4_WAIT_SPINS << 2);
}
// the same by a whole warp, with one answer for all of its lanes
__device__ __forceinline__ bool mbar_wait_item_warp(uint64_t* bar, uint32_t parity, volatile int* err, int site) {
  return __all_sync(0xffffffffu, mbar_wait_item(bar, parity, err, site));
}

// End of a kernel, by all of its threads behind the last barrier and before tensor memory is given back.  Where a wait has
// expired nothing has waited for the copies and products still under way: they get a millisecond (they take
// microseconds) before the CTA's memory is another's, and the site of the wait goes to the status word.
__device__ __forceinline__ void report_error(volatile int* err, int* status) {
  const int e = *err;
  if (e == 0) return;
#pragma unroll 1
  for (int i = 0; i < 1024; ++i) __nanosleep(1000);
  if (threadIdx.x == 0 && status != nullptr) atomicExch(status, e);
}
// The same as a function of its own, for the forward: the code in place made it slower where it never runs (D = 256 with
// a bias 2 %, S8192 0.5 %).  The call costs the backward and decode kernels a few spilled registers and the V
// projection 0.5 to 1.5 us (S1000 hidden 2048 10.8 -> 12.3).
static __device__ __noinline__ void report_error_call(volatile int* err, int* status) { report_error(err, status); }

// ------------------------------------------------------------------ cluster launch control
// A running CTA takes over the work of one that has not been launched yet: one thread asks (16 bytes arrive at
// `resp`, counted by `bar`), then any thread reads the answer.  After an answer without a CTA nothing may be asked again.
__device__ __forceinline__ void clc_request(void* resp, uint64_t* bar) {
  mbar_expect_tx(bar, 16);
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                   smem_u32(resp)),
               "r"(smem_u32(bar))
               : "memory");
}
// block index of the CTA taken over, or false where none was left
__device__ __forceinline__ bool clc_answer(const void* resp, int& x, int& y, int& z) {
  uint32_t got, bx = 0, by = 0, bz = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 r;\n\t"
      "ld.shared.b128 r, [%4];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, %2, %3, _}, r;\n\t}\n"
      : "=r"(got), "+r"(bx), "+r"(by), "+r"(bz)
      : "r"(smem_u32(resp))
      : "memory");
  x = (int)bx;
  y = (int)by;
  z = (int)bz;
  return got != 0;
}

// All threads of the cluster; `.aligned` wants the lanes of a warp together, whatever branches and loops lie behind them.
__device__ __forceinline__ void cluster_sync_all() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t saddr, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

__device__ __forceinline__ float ld_cluster_f32(uint32_t saddr, uint32_t rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// barrier among a subset of warps (id 1..15, nthreads multiple of 32)
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// generic-proxy writes (st.shared) -> visible to the async proxy (TMA / tcgen05 reads of smem)
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// shared-memory accesses by 32-bit shared address (keeps them out of the generic path)
__device__ __forceinline__ void sts_v2(uint32_t saddr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(saddr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void sts_b32(uint32_t saddr, uint32_t a) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(saddr), "r"(a) : "memory");
}
__device__ __forceinline__ void sts_f32(uint32_t saddr, float a) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(saddr), "f"(a) : "memory");
}
__device__ __forceinline__ float lds_f32(uint32_t saddr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(saddr) : "memory");
  return v;
}

// ------------------------------------------------------------------ TMA
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* m, uint64_t* bar, int c0,
                                            int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, "
      "%4, %5}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

__device__ __forceinline__ void tma_prefetch_map(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}

// Shared-memory box -> global memory, asynchronous in the issuing thread's bulk group.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* m, const void* src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void bulk_wait_read() {      // all but the last N stores have read their shared memory
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}

// L2 prefetch of a tensor-map box (no shared memory, no barrier).
__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap* m, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
// a run of bytes; address and size are multiples of 16
__device__ __forceinline__ void bulk_prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Per-thread asynchronous 4-byte global -> shared copy; src_bytes = 0 zero-fills.
__device__ __forceinline__ void cp_async_4(uint32_t saddr, const void* gptr, uint32_t src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(saddr), "l"(gptr), "r"(src_bytes)
               : "memory");
}
// The same with a hint that L2 should fetch the whole 128-byte line: for scattered small reads
// whose neighbours in the line are wanted a few tiles later (strided scale bytes).
__device__ __forceinline__ void cp_async_4_l2line(uint32_t saddr, const void* gptr, uint32_t src_bytes) {
  asm volatile("cp.async.ca.shared.global.L2::128B [%0], [%1], 4, %2;" ::"r"(saddr), "l"(gptr),
               "r"(src_bytes)
               : "memory");
}
// This thread's copies so far arrive on `bar` (once, counted among its expected arrivals) when they have landed.
__device__ __forceinline__ void cp_async_mbar_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ------------------------------------------------------------------ TMEM management
// Must be executed by one full warp. ncols: power of two in [32, 512].
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// ------------------------------------------------------------------ descriptors
// Shared-memory matrix descriptor, K-major operand, 16-byte units.
//   swizzle_code: 0 none, 2 = 128B, 4 = 64B, 6 = 32B.
//   sbo_bytes: distance between consecutive 8-row groups.
__host__ __device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr, uint32_t lbo_bytes,
                                                            uint32_t sbo_bytes,
                                                            uint32_t swizzle_code) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for sm_100
  d |= (uint64_t)(swizzle_code & 7) << 61;
  return d;
}

// Instruction descriptor (upper 32 bits of the i-desc operand) for
// kind::mxf4nvf4, e2m1 x e2m1, ue4m3 scales per 16, fp32 accumulate, both operands K-major.
__host__ __device__ __forceinline__ uint32_t make_idesc_nvfp4(uint32_t m, uint32_t n) {
  uint32_t d = 0;
  d |= 1u << 7;          // A format: e2m1
  d |= 1u << 10;         // B format: e2m1
  d |= (n >> 3) << 17;   // N / 8
  d |= 0u << 23;         // scale format: ue4m3
  d |= (m >> 4) << 24;   // M / 16
  return d;              // sf ids 0, K = 64
}

// D[tmem] (+)= A[smem] * B[smem]^T with block scales held in TMEM. One thread issues.
__device__ __forceinline__ void umma_nvfp4(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                           uint32_t idesc, uint32_t sfa_tmem, uint32_t sfb_tmem,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], "
      "p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem)
      : "memory");
}

// All tcgen05 async ops issued so far by this thread arrive (once) on `bar` when complete.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

// smem (32 rows x 16 bytes, rows 16 B apart) -> TMEM (32 lanes x 4 columns, replicated to the
// four 32-lane sub-partitions). One thread issues. Used for block-scale factors.
__device__ __forceinline__ void tmem_cp_32x128b_warpx4(uint32_t taddr, uint32_t saddr) {
  uint64_t desc = make_smem_desc(saddr, 0, 128, 0);
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(desc)
               : "memory");
}

// ------------------------------------------------------------------ TMEM <-> registers
// 32 lanes x 32 consecutive 32-bit columns; thread t of the warp gets lane (base_lane + t).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(
          taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
      "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
      "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
      "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
      "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// ------------------------------------------------------------------ operand layouts in smem
// Byte offset of (row, byte-in-row) inside a K-major tile whose rows are 64 bytes wide and
// stored with the 64-byte swizzle (8-row x 64 B = 512 B repeating pattern; tile base 512 B
// aligned): the 16-byte chunk index is XORed with bits [1,3) of the row.
__device__ __forceinline__ uint32_t sw64_offset(uint32_t row, uint32_t byte_in_row) {
  uint32_t chunk = byte_in_row >> 4;
  return row * 64u + (((chunk ^ (row >> 1)) & 3u) << 4) + (byte_in_row & 15u);
}
// Same for 128-byte rows with the 128-byte swizzle (8 x 128 B = 1 KB pattern, base 1 KB aligned).
__device__ __forceinline__ uint32_t sw128_offset(uint32_t row, uint32_t byte_in_row) {
  uint32_t chunk = byte_in_row >> 4;
  return row * 128u + (((chunk ^ row) & 7u) << 4) + (byte_in_row & 15u);
}
// Block-scale "atom" consumed by tcgen05.cp 32x128b.warpx4: 128 rows x 4 scale bytes (one
// K=64 MMA) stored as 32 x 16 B; row r, scale k sits at (r % 32) * 16 + (r / 32) * 4 + k.
__device__ __forceinline__ uint32_t sf_atom_offset(uint32_t row, uint32_t k) {
  return (row & 31u) * 16u + (row >> 5) * 4u + k;
}

}  // namespace nvfp4

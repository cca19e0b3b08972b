// Shared device-side helpers for the sm_100a kernels: mbarrier, TMA, tcgen05/TMEM wrappers,
// bounded waits and the kernel status word.
//
// Every wait in this library is bounded: a wait that runs out records a code in the status
// word handed to the kernel and returns false; the caller then leaves its role loop, joins the
// CTA-wide teardown, frees any TMEM it holds and returns.  Nothing here traps or spins forever.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

namespace pf {

// Codes written to a kernel status word (first error wins).
enum Status : int {
  PF_OK = 0,
  PF_ERR_TIMEOUT_FULL = 1,      // consumer waited on a full barrier
  PF_ERR_TIMEOUT_EMPTY = 2,     // producer waited on an empty barrier
  PF_ERR_TIMEOUT_TMEM_FULL = 3,
  PF_ERR_TIMEOUT_TMEM_EMPTY = 4,
  PF_ERR_TIMEOUT_PEER_FLAG = 5, // a flag owned by another GPU never arrived
  PF_ERR_BAD_ARG = 6,
};

// ~1 s at 1.9 GHz; waits in flight when a peer dies give up after this.
#ifndef PF_WAIT_CYCLES
#define PF_WAIT_CYCLES (2000000000ll)
#endif

// The status buffer handed to a kernel is int[PF_STATUS_WORDS]:
//   [0] first error code (0 = none), [1] wait limit in units of 1024 cycles (0 = PF_WAIT_CYCLES).
// The limit is a run-time value so that a caller (or a test that lets a wait run out on
// purpose) can shorten it without rebuilding the library.
constexpr int PF_STATUS_WORDS = 4;

__device__ __forceinline__ void report(int* status, int code) {
  if (status) atomicCAS(status, 0, code);
}

__device__ __forceinline__ long long wait_limit(const int* status) {
  if (status) {
    const int k = *reinterpret_cast<const volatile int*>(status + 1);
    if (k > 0) return static_cast<long long>(k) << 10;
  }
  return PF_WAIT_CYCLES;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred P;\n\t.reg .b32 R;\n\t"
      "elect.sync R|P, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}\n"
      : "=r"(pred));
  return pred != 0;
}

// Register split between warpgroups.  Every warp of the warpgroup executes it; the shares of all
// warpgroups add up to no more than the block was launched with.
template <int N> __device__ __forceinline__ void regs_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N> __device__ __forceinline__ void regs_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// Programmatic dependent launch: a kernel launched by `after` (below) may start when every CTA of the one
// before it in its stream has left, before that one's end is known everywhere, and calls this before it
// reads or writes anything that an earlier kernel may have to do with: it returns when all of those have
// completed and their results are visible.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// Called by a CTA after after_previous(): the next kernel may start as soon as every CTA has called it.  Only
// for a next kernel that needs nothing of this one; that one has a CTA call after_previous() before it
// leaves, so that whatever comes later finds both completed.
__device__ __forceinline__ void let_next_start() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ----------------------------------------------------------------------------- mbarrier
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
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// one look at the barrier, without waiting
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
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
// Bounded wait.  Returns false (after recording `code`) when the limit runs out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  // The limit lives in global memory and the clock costs a few cycles to read: both are looked
  // at only every 256 polls, so a wait that is satisfied soon pays for neither.
  long long t0 = 0, limit = 0;
  for (unsigned polls = 1; !mbar_try_wait(bar, parity); ++polls) {
    if ((polls & 255u) == 0) {
      if (limit == 0) { t0 = clock64(); limit = wait_limit(status); }
      else if (clock64() - t0 > limit) {
        report(status, code);
        return false;
      }
    }
  }
  return true;
}

// ----------------------------------------------------------------------------- TMA (no multicast)
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* m, uint64_t* bar,
                                            int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
      "{%3, %4}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0),
        "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* m, uint64_t* bar,
                                            int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
      "{%3, %4, %5}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0),
        "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* m, uint64_t* bar,
                                            int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
      "{%3, %4, %5, %6}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0),
        "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
// TMA stores (shared -> global), plain and with an fp32 add at the destination
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, const void* smem_src, int c0,
                                             int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               :
               : "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* m, const void* smem_src, int c0,
                                             int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               :
               : "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1),
                 "r"(c2), "r"(c3)
               : "memory");
}
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* m, const void* smem_src,
                                                  int c0, int c1) {
  asm volatile(
      "cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%2, %3}], [%1];"
      :
      : "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* m, const void* smem_src,
                                                  int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4, %5}], "
      "[%1];"
      :
      : "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2),
        "r"(c3)
      : "memory");
}
// plain (untiled) copy of `bytes` (a multiple of 16, both addresses 16-byte aligned)
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      :
      : "r"(smem_u32(smem_dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// per-thread asynchronous copies of 16 bytes, global -> shared
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
// all but the N most recently committed groups have landed (for the calling thread's copies)
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void tma_store_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// the staged source may be overwritten again
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
// all but the most recent group of stores have read their source
__device__ __forceinline__ void tma_store_wait_read_but_one() {
  asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
}
// the stores have completed
__device__ __forceinline__ void tma_store_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// generic-proxy writes to smem -> visible to the async proxy (tcgen05.mma / TMA store)
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ----------------------------------------------------------------------------- tcgen05 / TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
}
// the allocated base address, known to be the same for all lanes (every lane of the warp calls)
__device__ __forceinline__ uint32_t tmem_base_of(const uint32_t* smem_slot) {
  return __shfl_sync(0xffffffffu, *reinterpret_cast<const volatile uint32_t*>(smem_slot), 0);
}
__device__ __forceinline__ void tmem_relinquish() {
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
// arrive on an mbarrier once every tcgen05.mma issued so far by this thread has completed
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
// ----------------------------------------------------------------------------- CTA pairs
// Forms used by kernels launched as clusters of two CTAs that share one tcgen05.mma
// (cta_group::2): the even CTA of the pair issues the instruction, each CTA supplies its half of
// the operands from its own shared memory and receives its half of the accumulator rows in its
// own TMEM.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// every thread of every CTA of the cluster
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;"
               ::: "memory");
}
// shared::cluster address of `p` (an address in this CTA's shared memory) in CTA `rank`
__device__ __forceinline__ uint32_t mapa_u32(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait on a barrier that threads of the peer CTA arrive on
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, int* status,
                                                  int code) {
  if (mbar_try_wait_cluster(bar, parity)) return true;
  long long t0 = 0, limit = 0;
  for (unsigned polls = 1; !mbar_try_wait_cluster(bar, parity); ++polls) {
    if ((polls & 255u) == 0) {
      if (limit == 0) { t0 = clock64(); limit = wait_limit(status); }
      else if (clock64() - t0 > limit) {
        report(status, code);
        return false;
      }
    }
  }
  return true;
}
// TMA load into this CTA's shared memory whose completion bytes are counted on a barrier given
// by its shared::cluster address (the pair leader's).  No multicast.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* m,
                                                 uint32_t bar_cluster_addr, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster_addr),
        "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(void* smem_dst, const CUtensorMap* m,
                                                 uint32_t bar_cluster_addr, int c0, int c1, int c2,
                                                 int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster_addr),
        "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
// executed by the same warp of both CTAs of the pair
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
// arrive on the barrier at this shared-memory offset in every CTA of `cta_mask` once the MMAs
// issued so far by this thread have completed
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar, uint16_t cta_mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;" ::"r"(smem_u32(bar)),
      "h"(cta_mask)
      : "memory");
}
// Shared-memory matrix descriptor for tcgen05.mma (version 1 = Blackwell), 128-byte swizzle.
//   K-major operand : rows of 128 B (64 x 16-bit along K); 8 rows = one 1024 B swizzle atom;
//                     SBO = distance between 8-row groups; LBO unused (1).
//   MN-major operand: rows of 128 B (64 x 16-bit along M/N), one row per K index; 8 K-rows =
//                     one atom; SBO = distance between 8-K-row groups, LBO = distance between
//                     64-element blocks along M/N.
// The high word is constant (SBO 1024); the low one holds the start address and LBO, so that a step to
// the next slice of an operand is one 32-bit addition.
constexpr uint32_t TC_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t smem_addr, uint32_t lbo_bytes) {
  return ((smem_addr & 0x3FFFF) >> 4) | ((lbo_bytes >> 4) << 16);
}

// D[tmem] (+)= A * B, 16-bit inputs, fp32 accumulate.  One thread issues, chosen by elect_one() for
// the whole of its role, with operands that are the same for all lanes of its warp: the compiler then
// keeps them in uniform registers, where the instruction reads them.  a_lo, b_lo: the descriptors' low
// words.
// Cycles from one product to the next, M = 128, K = 16 (B200, 1 CTA, eight other warps busy), by the
// form of the issue: a lane chosen by `lane == 0` in a loop that builds 64-bit descriptors 109-124
// whatever N; a converged warp in which a predicate picks the lane 61-70; elected, unrolled: 32 at
// N = 64 with A in TMEM (what the arithmetic takes), 50 at N = 64 with A in shared memory (48 to
// fetch the operands), 66 at N = 128 (64).
__device__ __forceinline__ void tc_mma_f16(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo,
                                           uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 da, {%1, %5};\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}\n"
      :
      : "r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(TC_DESC_HI)
      : "memory");
}
// A operand from TMEM (attention: P stays on chip)
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo,
                                              uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t}\n"
      :
      : "r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(TC_DESC_HI)
      : "memory");
}
// D (256 rows over the two CTAs' TMEM) (+)= A (128 rows per CTA) * B (N/2 rows per CTA)
__device__ __forceinline__ void tc_mma_f16_pair(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo,
                                                uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 da, {%1, %5};\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n\t}\n"
      :
      : "r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(TC_DESC_HI)
      : "memory");
}

// 32 lanes x 32 columns of fp32: thread i of the warp receives 32 consecutive columns of TMEM
// lane (lane_base + i).  The warp may only touch lanes [32*(warp_id%4), +32).
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
// Wait for the TMEM loads in flight, with the loaded registers named as operands: a use of them is
// no memory access and could otherwise be scheduled ahead of the wait.
__device__ __forceinline__ void tmem_ld_wait_for(uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.wait::ld.sync.aligned;"
      : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
        "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]),
        "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]),
        "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]),
        "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
      :
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
        "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
        "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
        "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
        "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
        "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Instruction descriptor, kind::f16, fp32 accumulate.  fmt: 0 = fp16, 1 = bf16.
__host__ __device__ constexpr uint32_t make_idesc_f16(int m, int n, int fmt, int a_mn_major,
                                                      int b_mn_major) {
  return (1u << 4)                         // D format fp32
         | (uint32_t(fmt) << 7)            // A format
         | (uint32_t(fmt) << 10)           // B format
         | (uint32_t(a_mn_major) << 15)    // A major (0 = K)
         | (uint32_t(b_mn_major) << 16)    // B major (0 = K)
         | (uint32_t(n >> 3) << 17)        // N / 8
         | (uint32_t(m >> 4) << 24);       // M / 16
}

// ----------------------------------------------------------------------------- small math
__device__ __forceinline__ float gelu_erf(float x) {
  return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f));
}
__device__ __forceinline__ float dgelu_erf(float x) {
  const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
  const float pdf = 0.3989422804014327f * __expf(-0.5f * x * x);
  return cdf + x * pdf;
}
// pairs of fp32 values in one 64-bit register: one issue slot for two operations
__device__ __forceinline__ uint64_t f2_pack(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
// two fp32 fused multiply-adds in one issue slot
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// erf-GELU and its derivative for fused GEMM epilogues, two values at a time: erf through the
// five-term rational approximation 1 - (a1 t + ... + a5 t^5) exp(-z^2), t = 1 / (1 + p z)
// (Abramowitz and Stegun 7.1.26, absolute error 1.5e-7), which costs two special-function
// instructions per value and nine packed ones per pair; gelu and gelu' are exact to 4e-7 absolute.
// With y = 0.5 poly exp(-x^2 / 2) >= 0, Phi(x) = y for x < 0 and 1 - y for x >= 0, so that
// gelu(x) = max(x, 0) - |x| y.  Phi is selected and not folded into 0.5 + sign(x) (0.5 - y): below -4 that
// would leave a few bits of y, and gelu' with a relative error of up to 3e-2 for 1.5e-4.
// Returns -y for |x| (`ax`) and leaves exp(-x^2 / 2) in `e`.  Every step rounds where the form for one
// value did, as does the last product of gelu: folding 1 / sqrt(2) into p and into the exponent, and that
// product into the sum, saves two instructions per pair and turns last bits, which twelve layers of
// 16-bit roundings carry on.
__device__ __forceinline__ uint64_t gelu_neg_tail2(uint64_t ax, uint64_t& e) {
  const uint64_t z = mul2(ax, f2_pack(0.70710678118654752f, 0.70710678118654752f));
  float d0, d1, q0, q1;
  f2_unpack(fma2(z, f2_pack(0.3275911f, 0.3275911f), f2_pack(1.f, 1.f)), d0, d1);
  f2_unpack(mul2(mul2(z, z), f2_pack(-1.4426950408889634f, -1.4426950408889634f)), q0, q1);
  const uint64_t t = f2_pack(rcp_approx(d0), rcp_approx(d1));
  e = f2_pack(exp2f(q0), exp2f(q1));
  uint64_t poly = fma2(t, f2_pack(-0.5f * 1.061405429f, -0.5f * 1.061405429f),
                       f2_pack(0.5f * 1.453152027f, 0.5f * 1.453152027f));
  poly = fma2(t, poly, f2_pack(-0.5f * 1.421413741f, -0.5f * 1.421413741f));
  poly = fma2(t, poly, f2_pack(0.5f * 0.284496736f, 0.5f * 0.284496736f));
  poly = fma2(t, poly, f2_pack(-0.5f * 0.254829592f, -0.5f * 0.254829592f));
  return mul2(mul2(poly, t), e);
}
// (a, b) -> gelu of both
__device__ __forceinline__ void gelu_erf_fast2(float& a, float& b) {
  uint64_t e;
  const uint64_t ax = f2_pack(fabsf(a), fabsf(b));
  float na, nb;                              // -|x| y
  f2_unpack(mul2(ax, gelu_neg_tail2(ax, e)), na, nb);
  // not packed: a packed product and the packed sum after it come out as one operation
  a = __fadd_rn(fmaxf(a, 0.f), na);
  b = __fadd_rn(fmaxf(b, 0.f), nb);
}
// (a, b) *= gelu' of (x, y)
__device__ __forceinline__ void dgelu_erf_fast2(float& a, float& b, float x, float y) {
  uint64_t e;
  const uint64_t ny = gelu_neg_tail2(f2_pack(fabsf(x), fabsf(y)), e);
  float y0, y1, c0, c1;
  f2_unpack(ny, y0, y1);
  f2_unpack(add2(ny, f2_pack(1.f, 1.f)), c0, c1);
  const uint64_t cdf = f2_pack(x >= 0.f ? c0 : -y0, y >= 0.f ? c1 : -y1);
  const uint64_t pdf_x = mul2(f2_pack(x, y), f2_pack(0.3989422804014327f, 0.3989422804014327f));
  f2_unpack(mul2(f2_pack(a, b), fma2(pdf_x, e, cdf)), a, b);
}
__device__ __forceinline__ float gelu_tanh(float x) {
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  return 0.5f * x * (1.0f + tanhf(u));
}
__device__ __forceinline__ float dgelu_tanh(float x) {
  const float x2 = x * x;
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x2);
  const float t = tanhf(u);
  const float du = 0.7978845608028654f * (1.0f + 3.0f * 0.044715f * x2);
  return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * du;
}
__device__ __forceinline__ float silu(float x) { return x / (1.0f + __expf(-x)); }
__device__ __forceinline__ float dsilu(float x) {
  const float s = 1.0f / (1.0f + __expf(-x));
  return s * (1.0f + x * (1.0f - s));
}

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) {
  return __bfloat162float(v);
}
template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

}  // namespace pf

// dtype codes shared with the Python side
#define PF_F32 0
#define PF_F16 1
#define PF_BF16 2

#define PF_API extern "C" __attribute__((visibility("default")))

// `after(kernel, grid, block, smem, stream)(arguments)` launches a kernel that calls after_previous().
// The launch and the kernel's set-up then lie under the end of the one before, some 2 us of each.  As a
// caller sees them, without and with: attention [24, 257, 16, 88] 155 -> 146.5 us (four launches), GroupNorm
// [4, 128, 128, 320] 103 -> 89 (six), a convolution 351 -> 341 (eight), forward and backward each.  No kernel
// lets one that depends on it start sooner: CTAs that wait on an SM take its place from others (171, 95 and
// 345).
template <typename... P>
struct LaunchAfter {
  void (*kernel)(P...);
  cudaLaunchConfig_t cfg;
  cudaError_t operator()(const P&... args) {
    cudaLaunchAttribute attr[2];
    int n = 0;
    for (; n < (int)cfg.numAttrs; ++n) attr[n] = cfg.attrs[n];       // a cluster's size
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = n + 1;
    void* list[] = {const_cast<void*>(static_cast<const void*>(&args))...};
    return cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(kernel), list);
  }
};
template <typename... P>
inline LaunchAfter<P...> after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                               cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  return {kernel, cfg};
}

// Whether operands that a kernel reads or writes 16 bytes at a time lie on 16 bytes (one that is left out
// does): an access that does not is a fault which ends the context, so entry points refuse it (-2).
template <typename... P>
inline bool on_vectors(const P*... operands) {
  return ((reinterpret_cast<uintptr_t>(operands) | ...) & 15) == 0;
}

#define PF_CHECK_LAUNCH()                            \
  do {                                               \
    cudaError_t e__ = cudaGetLastError();            \
    if (e__ != cudaSuccess) return static_cast<int>(e__); \
  } while (0)

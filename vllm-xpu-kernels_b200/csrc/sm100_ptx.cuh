// Thin inline-PTX wrappers for the sm_100a features the grouped GEMM uses:
// mbarrier, TMA tiled loads (cp.async.bulk.tensor; every load lands in the shared
// memory of the CTA that issued it), tensor memory allocation, tcgen05.mma /
// commit / ld (one CTA, or a pair of CTAs of a cluster on one tile) and the
// shared-memory and instruction descriptors they take.  Every spin-wait on an
// mbarrier here is bounded.
#pragma once

#include <cuda.h>
#include <stdint.h>

namespace b200moe {
namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// ---- mbarrier ---------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
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

// Waits for the phase with `parity` to complete, for at most about
// `kWaitBudgetCycles` clock cycles or until `*abort_flag` becomes non-zero.
// Returns false (and raises the flag) when it gave up.
constexpr long long kWaitBudgetCycles = 2000000000LL;  // roughly one second
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          long long budget_cycles = kWaitBudgetCycles) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 0xff) == 0) {
      if (*abort_flag != 0) return false;
      if (clock64() - t0 > budget_cycles) {
        *abort_flag = 1;
        return false;
      }
    }
  }
  return true;
}

// The wait of the producer and issuer loops, which are single threads whose instruction chain
// bounds a CTA's streaming rate: barriers are 32-bit shared addresses and only the first poll is
// inline (measured on a loop of one wait, one expect_tx and one load: 198 instead of 378 cycles).
// Same budget and abort rules as mbar_wait.
__device__ __forceinline__ bool mbar_try_wait_s(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// One look, without the suspension a try_wait may take.
__device__ __forceinline__ bool mbar_test_wait_s(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
static __device__ __noinline__ bool mbar_wait_rest(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  const long long t0 = clock64();
  while (!mbar_try_wait_s(bar, parity)) {   // (paced, see below)
    if (*abort_flag != 0) return false;
    if (clock64() - t0 > kWaitBudgetCycles) {
      *abort_flag = 1;
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ bool mbar_wait_s(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return mbar_try_wait_s(bar, parity) || mbar_wait_rest(bar, parity, abort_flag);
}
// The same for waits that a role with a queue ahead of it sits out (producers for a free stage, preparers and
// converters for theirs): without a call, whose way back stood between the phase's end and the next load, and with both
// bounds looked at after every poll, which makes polls rarer: they take turns in one unit with the arrivals and
// waits of the roles that are behind (eight polls in a row without anything between them cost the int4 kernel 4 %, the
// MXFP4 one 2 %; a sleep between them 1 to 2 %).  Layer calls that follow one another, call and counter / so, us: DeepSeek at
// 8192 tokens 4929 / 4737, one of its 8 ranks at 1024 tokens 280.5 / 275.9, qwen3 at 3001 tokens 307.6 / 301.1, gpt-oss at 2048
// tokens 764 / 751, at 128 tokens 391.8 / 389.9 (no difference: runs of one side differ by 0.7 %; in bursts of 20 ms after
// a rest 342 / 337), int4 Mixtral at 33 tokens 231.5 / 230.0.
namespace paced {
__device__ __forceinline__ bool mbar_wait_s(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait_s(bar, parity)) return true;
  const long long t0 = clock64();
#pragma unroll 1
  while (!mbar_try_wait_s(bar, parity)) {
    if (*abort_flag != 0) return false;
    if (clock64() - t0 > kWaitBudgetCycles) {
      *abort_flag = 1;
      return false;
    }
  }
  return true;
}
}  // namespace paced
// The same without a call, for warps whose registers are full.
__device__ __forceinline__ bool mbar_wait_inline_s(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait_s(bar, parity)) return true;
  const long long t0 = clock64();
  uint32_t spins = 0;
#pragma unroll 1
  while (!mbar_try_wait_s(bar, parity)) {
    if ((++spins & 0xff) == 0) {
      if (*abort_flag != 0) return false;
      if (clock64() - t0 > kWaitBudgetCycles) {
        *abort_flag = 1;
        return false;
      }
    }
  }
  return true;
}
// The same without a call and for warps whose registers are full: one register for the time, the abort flag
// by its shared address.
__device__ __forceinline__ bool mbar_wait_lean(uint32_t bar, uint32_t parity, uint32_t abort_flag) {
  if (mbar_try_wait_s(bar, parity)) return true;
  const uint32_t t0 = (uint32_t)clock();
  uint32_t spins = 0;
#pragma unroll 1
  while (!mbar_try_wait_s(bar, parity)) {
    if ((++spins & 0xff) != 0) continue;
    uint32_t aborted;
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(aborted) : "r"(abort_flag) : "memory");
    if (aborted != 0) return false;
    if ((uint32_t)clock() - t0 > (uint32_t)kWaitBudgetCycles) {
      asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(abort_flag), "r"(1) : "memory");
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ void mbar_arrive_s(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// ... by the lanes for which `p` holds, without a branch
__device__ __forceinline__ void mbar_arrive_if(uint32_t bar, bool p) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\t@q mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar),
               "r"((uint32_t)p)
               : "memory");
}
// ... and, where `also` holds too, on a second barrier
__device__ __forceinline__ void mbar_arrive_if(uint32_t bar, bool p, uint32_t second, bool also) {
  asm volatile("{\n\t.reg .pred q, t;\n\tsetp.ne.u32 q, %2, 0;\n\tsetp.ne.and.u32 t, %3, 0, q;\n\t"
               "@q mbarrier.arrive.shared::cta.b64 _, [%0];\n\t@t mbarrier.arrive.shared::cta.b64 _, [%1];\n\t}" ::"r"(bar),
               "r"(second), "r"((uint32_t)p), "r"((uint32_t)also)
               : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_s(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// True in one lane of a converged warp.  Code under it issues TMA and MMA instructions about twice
// as fast as under `lane == 0`: the compiler knows that a single lane runs it.
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
  return one != 0;
}

// Warp-level wait: lane 0 polls (sleeping `sleep_ns` between polls when non-zero),
// the other lanes wait at the warp barrier, which also orders their later reads
// after the barrier's completion.  Keeps the polling traffic of long waits off
// the shared-memory pipeline that other warps need.  Same budget and abort rules
// as mbar_wait; every lane gets the result.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity,
                                               volatile int* abort_flag, uint32_t sleep_ns) {
  bool ok = true;
  if ((threadIdx.x & 31) == 0 && !mbar_try_wait(bar, parity)) {
    const long long t0 = clock64();
    uint32_t spins = 0;
    while (!mbar_try_wait(bar, parity)) {
      if (sleep_ns) __nanosleep(sleep_ns);
      if ((++spins & 0x3f) == 0) {
        if (*abort_flag != 0) { ok = false; break; }
        if (clock64() - t0 > kWaitBudgetCycles) { *abort_flag = 1; ok = false; break; }
      }
    }
  }
  ok = __shfl_sync(0xffffffffu, ok, 0);
  __syncwarp();
  return ok;
}

// ---- TMA ---------------------------------------------------------------------
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// (Destination and barrier are 32-bit shared addresses.)
__device__ __forceinline__ void tma_load_2d_s(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_s(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                              int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

// Brings the box into L2 only.
__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap* map, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global [%0, {%1, %2, %3}];" ::"l"(reinterpret_cast<uint64_t>(map)), "r"(c0),
               "r"(c1), "r"(c2)
               : "memory");
}

// Tiled store from this CTA's shared memory; the rows the box covers all belong to the caller.  The thread
// that issues it commits a group, and waits for it before the memory is written again or the CTA ends.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// All groups of this thread have read their shared memory / are complete.
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ---- CTA pairs (a cluster of two CTAs working on one tcgen05.mma tile) ----------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_id_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_count_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
  return r;
}
// All threads of all CTAs of the cluster.  Not bounded: call it only where every thread
// of both CTAs arrives after bounded work.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The shared::cluster address of `addr` (a shared address of this CTA) in CTA `rank`.
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Arrival on a barrier of any CTA of the cluster.  Relaxed: the callers hand back tensor
// memory whose reads tcgen05.wait::ld has already completed, nothing else has to be visible
// (with .release.cluster every arrival costs a cluster-scope fence: measured 2x on a loop
// that arrives once per K block).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// The same with release semantics at cluster scope: what this thread (and, through a preceding
// __syncwarp, its warp) wrote to the other CTA's shared memory is visible to whoever acquires
// the barrier's phase.
__device__ __forceinline__ void mbar_arrive_cluster_release(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Bounded wait on a barrier of this CTA whose phase another CTA of the cluster completes
// (acquire at cluster scope: that CTA's stores into this CTA's shared memory are visible after).
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  const uint32_t addr = smem_u32(bar);
  auto try_wait = [&]() {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    return ok != 0;
  };
  if (try_wait()) return true;
  const long long t0 = clock64();
  uint32_t spins = 0;
  while (!try_wait()) {
    if ((++spins & 0xff) == 0) {
      if (*abort_flag != 0) return false;
      if (clock64() - t0 > kWaitBudgetCycles) {
        *abort_flag = 1;
        return false;
      }
    }
  }
  return true;
}
// 16-byte store into the shared memory of any CTA of the cluster.
__device__ __forceinline__ void st_cluster_v4(uint32_t cluster_addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "f"(a), "f"(b), "f"(c), "f"(d)
               : "memory");
}
// Tiled loads of a CTA pair: the data lands in the issuing CTA's shared memory, the bytes
// are counted on `bar_cluster_addr`, which may be the other CTA's barrier.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster_addr,
                                                 int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster_addr,
                                                 int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

// ---- tensor memory -------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
// The same for a CTA pair: the same warp of both CTAs executes each of them.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// 32 lanes x 32 consecutive 32-bit columns: thread i gets lane (base lane + i).
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr)
      : "memory");
}

// Waits for all of this thread's tcgen05.ld.  The registers they filled are operands of a statement behind
// the wait (it emits nothing; volatile asm statements keep their order), so that no use of them is scheduled
// ahead of it.
template <int... N>
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&...r)[N]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  auto pin = [](auto& a) {
#pragma unroll
    for (uint32_t& x : a) asm volatile("" : "+r"(x));
  };
  (pin(r), ...);
}
// Register re-balancing between the warpgroups of a CTA (every warp of a warpgroup
// executes the same one): dec gives registers back to the CTA's pool, inc waits until
// the pool holds enough and takes them.
template <int kRegs>
__device__ __forceinline__ void setmaxnreg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs));
}
template <int kRegs>
__device__ __forceinline__ void setmaxnreg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs));
}
// 32 lanes x N consecutive 32-bit columns written from registers: thread i
// writes lane (base lane + i).
__device__ __forceinline__ void tmem_st_32x4(uint32_t taddr, uint32_t r0, uint32_t r1, uint32_t r2,
                                             uint32_t r3) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(r0),
               "r"(r1), "r"(r2), "r"(r3)
               : "memory");
}
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
        "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// 32 bytes of one thread to a 32-byte aligned global address.
__device__ __forceinline__ void stg256(void* to, const uint32_t (&w)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(to), "r"(w[0]), "r"(w[1]), "r"(w[2]),
               "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

// ---- UMMA ------------------------------------------------------------------------
// Shared-memory matrix descriptor, 128-byte swizzle, sm_100 version bit set.
// lbo / sbo in bytes (16-byte units once encoded).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes,
                                                   uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3fff);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3fff) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3fff) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of sm_100
  d |= (uint64_t)2 << 61;  // SWIZZLE_128B
  return d;
}

// The same without a swizzle: rows of 16 bytes, eight rows (one 128-byte core matrix) after
// another, core matrices `sbo_bytes` apart.
__device__ __forceinline__ uint64_t make_smem_desc_plain(uint32_t smem_addr, uint32_t sbo_bytes) {
  return (uint64_t)((smem_addr >> 4) & 0x3fff) | ((uint64_t)((sbo_bytes >> 4) & 0x3fff) << 32) | ((uint64_t)1 << 46);
}

// Instruction descriptor of tcgen05.mma kind::f16 / kind::f8f6f4, fp32 accumulate.
// fmt: kind::f16 -> 0 = f16, 1 = bf16; kind::f8f6f4 -> 0 = e4m3, 1 = e5m2.
// major: 0 = K-major, 1 = MN-major.
__host__ __device__ constexpr uint32_t make_idesc(uint32_t a_fmt, uint32_t b_fmt, uint32_t a_major,
                                                  uint32_t b_major, uint32_t M, uint32_t N) {
  return (1u << 4) | (a_fmt << 7) | (b_fmt << 10) | (a_major << 15) | (b_major << 16) |
         ((N >> 3) << 17) | ((M >> 4) << 24);
}

// Instruction descriptor of tcgen05.mma kind::mxf8f6f4.block_scale with e8m0
// scales: a_fmt / b_fmt 0 = e4m3, 1 = e5m2, 3 = e2m3, 4 = e3m2, 5 = e2m1; both
// operands K-major; fp32 accumulate.  The scale byte (0..3) of the 32-bit scale
// column each operand uses is OR-ed in per instruction: a at bit 29, b at bit 4.
__host__ __device__ constexpr uint32_t make_idesc_mx(uint32_t a_fmt, uint32_t b_fmt, uint32_t M,
                                                     uint32_t N) {
  return (a_fmt << 7) | (b_fmt << 10) | ((N >> 3) << 17) | (1u << 23) | ((M >> 4) << 24);
}
// Block-scaled form: D[tmem_d] (+)= (A * 2^(sfa-127)) * (B * 2^(sfb-127)) over K = 32; sfa / sfb
// are tensor-memory addresses of the scale columns (one byte per row, replicated in the four
// lane quarters).  Issued by one thread (elect_one), like umma_commit.
//
// One 128-wide K block in one statement: the block's scale chunks are copied from shared to tensor
// memory (tcgen05.cp 32x128b.warpx4: 32 rows of 16 bytes -> four columns, replicated in the four
// lane quarters; the weight rows' to column sf, the tokens' kTokChunks chunks to the columns after
// them), then the four K = 32 instructions run on scale bytes 0..3 of those columns.  kWStep:
// 16-byte units between the K steps of the weight operand (the tokens' are 32 bytes apart).
// Descriptors come as halves, of which only the lower ones (addresses) differ between blocks: 64-bit
// additions cost the issuing thread 20 cycles a K block.
template <int kTokChunks, int kWStep>
__device__ __forceinline__ void umma_mx_block(uint32_t tmem_d, uint32_t wdesc, uint32_t w_hi, uint32_t adesc, uint32_t a_hi,
                                              uint32_t idesc, uint32_t accumulate, uint32_t sf, uint32_t sfw_desc,
                                              uint32_t sfa_desc, uint32_t sf_hi) {
#define B200_MX_MMA4                                                                                                   \
      "mov.b64 w0, {%1, %2};\n\tmov.b64 a0, {%3, %4};\n\t"                                                             \
      "add.u32 x1, %1, %11;\n\tadd.u32 x2, %1, %12;\n\tadd.u32 x3, %1, %13;\n\t"                                      \
      "add.u32 y1, %3, 2;\n\tadd.u32 y2, %3, 4;\n\tadd.u32 y3, %3, 6;\n\t"                                            \
      "mov.b64 w1, {x1, %2};\n\tmov.b64 w2, {x2, %2};\n\tmov.b64 w3, {x3, %2};\n\t"                                   \
      "mov.b64 a1, {y1, %4};\n\tmov.b64 a2, {y2, %4};\n\tmov.b64 a3, {y3, %4};\n\t"                                   \
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], w0, a0, %5, [%7], [t], pa;\n\t"                       \
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], w1, a1, i1, [%7], [t], 1;\n\t"                        \
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], w2, a2, i2, [%7], [t], 1;\n\t"                        \
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], w3, a3, i3, [%7], [t], 1;\n\t}"
#define B200_MX_HEAD                                                                                                   \
      "{\n\t.reg .pred pa;\n\t.reg .b32 t, t2, c2, i1, i2, i3, x1, x2, x3, y1, y2, y3;\n\t"                           \
      ".reg .b64 s0, s1, s2, w0, w1, w2, w3, a0, a1, a2, a3;\n\t"                                                      \
      "setp.ne.b32 pa, %6, 0;\n\tadd.u32 t, %7, 4;\n\t"                                                                \
      "or.b32 i1, %5, 0x20000010;\n\tor.b32 i2, %5, 0x40000020;\n\tor.b32 i3, %5, 0x60000030;\n\t"                    \
      "mov.b64 s0, {%8, %10};\n\tmov.b64 s1, {%9, %10};\n\t"                                                          \
      "tcgen05.cp.cta_group::1.32x128b.warpx4 [%7], s0;\n\t"                                                           \
      "tcgen05.cp.cta_group::1.32x128b.warpx4 [t], s1;\n\t"
  if (kTokChunks == 1) {
    asm volatile(B200_MX_HEAD B200_MX_MMA4
                 ::"r"(tmem_d), "r"(wdesc), "r"(w_hi), "r"(adesc), "r"(a_hi), "r"(idesc), "r"(accumulate), "r"(sf),
                 "r"(sfw_desc), "r"(sfa_desc), "r"(sf_hi), "n"(kWStep), "n"(2 * kWStep), "n"(3 * kWStep)
                 : "memory");
  } else {
    asm volatile(B200_MX_HEAD
                 "add.u32 t2, %7, 8;\n\tadd.u32 c2, %9, 32;\n\tmov.b64 s2, {c2, %10};\n\t"
                 "tcgen05.cp.cta_group::1.32x128b.warpx4 [t2], s2;\n\t" B200_MX_MMA4
                 ::"r"(tmem_d), "r"(wdesc), "r"(w_hi), "r"(adesc), "r"(a_hi), "r"(idesc), "r"(accumulate), "r"(sf),
                 "r"(sfw_desc), "r"(sfa_desc), "r"(sf_hi), "n"(kWStep), "n"(2 * kWStep), "n"(3 * kWStep)
                 : "memory");
  }
#undef B200_MX_MMA4
#undef B200_MX_HEAD
}
// The four K = 32-byte instructions of one 128-byte-wide K block, issued by one thread (elect_one):
// both descriptors advance by an addition, only the first instruction may overwrite D.  kAStep and
// kBStep: 16-byte units between the K steps of the two operands.
template <bool kFp8, int kAStep, int kBStep>
__device__ __forceinline__ void umma_block(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
#define B200_UMMA4(KIND)                                                                                \
  asm volatile(                                                                                          \
      "{\n\t.reg .pred pa;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\tsetp.ne.b32 pa, %4, 0;\n\t"                \
      "add.u64 a1, %1, %5;\n\tadd.u64 a2, %1, %6;\n\tadd.u64 a3, %1, %7;\n\t"                            \
      "add.u64 b1, %2, %8;\n\tadd.u64 b2, %2, %9;\n\tadd.u64 b3, %2, %10;\n\t"                           \
      "tcgen05.mma.cta_group::1.kind::" KIND " [%0], %1, %2, %3, pa;\n\t"                                \
      "tcgen05.mma.cta_group::1.kind::" KIND " [%0], a1, b1, %3, 1;\n\t"                                 \
      "tcgen05.mma.cta_group::1.kind::" KIND " [%0], a2, b2, %3, 1;\n\t"                                 \
      "tcgen05.mma.cta_group::1.kind::" KIND " [%0], a3, b3, %3, 1;\n\t}"                                \
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "n"(kAStep), "n"(2 * kAStep),  \
        "n"(3 * kAStep), "n"(kBStep), "n"(2 * kBStep), "n"(3 * kBStep)                                    \
      : "memory")
  if (kFp8) B200_UMMA4("f8f6f4");
  else B200_UMMA4("f16");
#undef B200_UMMA4
}
// A 512-byte scale chunk from shared to tensor memory, as in umma_mx_block.
__device__ __forceinline__ void tmem_cp_scales(uint32_t taddr, uint64_t desc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(desc) : "memory");
}
// umma_mx_block's four instructions with the weights in tensor memory (eight columns per K step).
__device__ __forceinline__ void umma_mx_block_ts(uint32_t tmem_d, uint32_t tmem_w, uint32_t adesc, uint32_t a_hi,
                                                 uint32_t idesc, uint32_t accumulate, uint32_t sfw, uint32_t sfa) {
  asm volatile(
      "{\n\t.reg .pred pa;\n\t.reg .b32 w1, w2, w3, i1, i2, i3, y1, y2, y3;\n\t.reg .b64 a0, a1, a2, a3;\n\t"
      "setp.ne.b32 pa, %7, 0;\n\t"
      "add.u32 w1, %1, 8;\n\tadd.u32 w2, %1, 16;\n\tadd.u32 w3, %1, 24;\n\t"
      "add.u32 y1, %2, 2;\n\tadd.u32 y2, %2, 4;\n\tadd.u32 y3, %2, 6;\n\t"
      "mov.b64 a0, {%2, %3};\n\tmov.b64 a1, {y1, %3};\n\tmov.b64 a2, {y2, %3};\n\tmov.b64 a3, {y3, %3};\n\t"
      "or.b32 i1, %4, 0x20000010;\n\tor.b32 i2, %4, 0x40000020;\n\tor.b32 i3, %4, 0x60000030;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], [%1], a0, %4, [%5], [%6], pa;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], [w1], a1, i1, [%5], [%6], 1;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], [w2], a2, i2, [%5], [%6], 1;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], [w3], a3, i3, [%5], [%6], 1;\n\t}"
      ::"r"(tmem_d), "r"(tmem_w), "r"(adesc), "r"(a_hi), "r"(idesc), "r"(sfw), "r"(sfa), "r"(accumulate)
      : "memory");
}
// Waits for this thread's tcgen05.ld and makes `r` depend on it.
__device__ __forceinline__ void tmem_wait_ld_one(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                 "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]),
                 "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]),
                 "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}
// acc[i] += v[i] * s for 32 values, two per instruction (each rounded as fmaf rounds it).
__device__ __forceinline__ void fma_f32x2(float2* acc, const uint32_t (&v)[32], float s) {
#pragma unroll
  for (int i = 0; i < 16; ++i)
    asm volatile("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmov.b64 c, {%0, %1};\n\t"
        "fma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "+f"(acc[i].x), "+f"(acc[i].y)
        : "r"(v[2 * i]), "r"(v[2 * i + 1]), "f"(s));
}
// acc += (v + m) * s for two values at once, each rounded as an addition and an fmaf round it.
__device__ __forceinline__ void add_fma_f32x2(float2& acc, uint32_t v0, uint32_t v1, float m0, float m1, float s) {
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tadd.rn.f32x2 a, a, b;\n\t"
      "mov.b64 b, {%6, %6};\n\tmov.b64 c, {%0, %1};\n\tfma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
      : "+f"(acc.x), "+f"(acc.y)
      : "r"(v0), "r"(v1), "f"(m0), "f"(m1), "f"(s));
}
// umma_block's four kind::f16 instructions with the 128-row operand in tensor memory (eight columns per
// K step, the other operand 32 bytes).
__device__ __forceinline__ void umma_f16_block_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                                  uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred pa;\n\t.reg .b32 a1, a2, a3;\n\t.reg .b64 b1, b2, b3;\n\tsetp.ne.b32 pa, %4, 0;\n\t"
      "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
      "add.u64 b1, %2, 2;\n\tadd.u64 b2, %2, 4;\n\tadd.u64 b3, %2, 6;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, pa;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, 1;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, 1;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, 1;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// A commit makes the barrier receive one arrival when all tcgen05 operations issued so far by this
// thread have completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// kind::f16 issued by the even CTA of a pair for both: M = 256 (128 rows of A and of D per CTA), each
// CTA holds N / 2 rows of B at the same shared-memory offsets, D at the same tensor-memory address in
// both.  One K block as in umma_block.
template <int kAStep, int kBStep>
__device__ __forceinline__ void umma_f16_pair_block(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                                    uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred pa;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\tsetp.ne.b32 pa, %4, 0;\n\t"
      "add.u64 a1, %1, %5;\n\tadd.u64 a2, %1, %6;\n\tadd.u64 a3, %1, %7;\n\t"
      "add.u64 b1, %2, %8;\n\tadd.u64 b2, %2, %9;\n\tadd.u64 b3, %2, %10;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, pa;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], a1, b1, %3, 1;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], a2, b2, %3, 1;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], a3, b3, %3, 1;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "n"(kAStep), "n"(2 * kAStep),
        "n"(3 * kAStep), "n"(kBStep), "n"(2 * kBStep), "n"(3 * kBStep)
      : "memory");
}
// One arrival on the barrier at `bar`'s offset in both CTAs of the pair once the pair's MMAs
// issued so far have completed.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .b16 m;\n\tmov.b16 m, 3;\n\t"
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n\t}"
      ::"r"(bar)
      : "memory");
}

// Explicit shared-space accesses (32-bit shared addresses): pointers derived
// from the re-aligned dynamic shared memory base are otherwise treated as
// generic and take the slower generic load/store path.
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void sts16(uint32_t addr, uint16_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"(v) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void sts32f(uint32_t addr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ float lds32f(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ float4 lds128f(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}

__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t lds8(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}

// 16-byte asynchronous copy global -> shared; only the first `src_bytes` are read,
// the rest of the 16 bytes is zero-filled.  Both addresses 16-byte aligned.
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes)
               : "memory");
}
// One arrival on `bar` once all cp.async copies this thread issued so far have
// landed (the arrival is part of the barrier's expected count).
__device__ __forceinline__ void cp_async_mbar_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

}  // namespace ptx
}  // namespace b200moe

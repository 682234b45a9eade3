// Thin inline-PTX wrappers for the sm_100a features the grouped GEMM uses:
// mbarrier (with bounded waits), TMA tiled loads, tcgen05 MMA / TMEM.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace syfi {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ------------------------------------------------- programmatic dependent launch
// Blocks until the kernel this one depends on has completed and its writes are visible
// (no-op when the kernel was launched without the programmatic-serialization attribute).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel in the stream be scheduled once every CTA has executed this (or exited).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
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

// Waits for the phase with the given parity, but never for ever: after
// `limit_cycles` SM clocks, or as soon as another thread of the CTA raised
// `*abort_flag`, it gives up, raises the flag itself and returns false.  The
// caller then leaves its role loop; the kernel tail records the failure in
// global memory and still releases tensor memory.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                  int code, long long limit_cycles = (1ll << 32)) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag != 0) return false;
    if (clock64() - t0 > limit_cycles) {
      *abort_flag = code;
      return false;
    }
  }
}

// The same for the warps that read tensor memory.  Each lane asks for itself and the lanes may disagree about a wait that
// runs out, but the loads of tensor memory and the shuffles behind them need all 32: so a failed lane clears `ok`, stays in
// its loop without waiting any more, and the warp votes on `ok` behind the loop.  What it costs lies in the warp's
// instructions (us per call at 4096 and 8192 tokens; lanes that leave the loop: 501.1, 845.7): this form 502.6 and 846.0, a
// call of mbar_wait_bounded behind the first look 504.0 and 849.4, `ok` asked before each wait and arrival 1 % more.
__device__ __forceinline__ void mbar_wait_or_clear(bool& ok, uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                   int code, long long limit_cycles) {
  if (mbar_try_wait(bar, parity)) return;
  const long long t0 = clock64();
  while (ok && !mbar_try_wait(bar, parity)) {
    if (*abort_flag != 0) {
      ok = false;
    } else if (clock64() - t0 > limit_cycles) {
      *abort_flag = code;
      ok = false;
    }
  }
}

// Waits for copies or MMAs that are already on their way.  They need nobody's help, so no abort flag ends this wait, which is
// for a CTA that gave up: its memory must not be handed to the next CTA with a write still coming.  Bounded all the same.
__device__ __forceinline__ void mbar_wait_landed(uint64_t* bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity) && clock64() - t0 < (1ll << 28)) {}
}

// Cross-CTA hand-off through a counter in global memory: the writers' data stores happen before the
// release increment, the reader's acquire load happens before its dependent loads.  The proxy fence
// orders generic-proxy accesses against async-proxy ones (TMA), which otherwise have no mutual order.
__device__ __forceinline__ void fence_proxy_async_all() {
  asm volatile("fence.proxy.async;" ::: "memory");
}
__device__ __forceinline__ void red_release_gpu_add(int* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_release_gpu(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// ----------------------------------------------------------------------- TMA
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_normal() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// 2-D tiled load, global -> this CTA's shared memory, completion on an mbarrier.
// x is the innermost (contiguous) coordinate; x * element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y,
                                            uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y),
        "l"(policy)
      : "memory");
}

// The same from a stack of matrices (3-D tensor map).
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z,
                                            uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4, %5}], [%2], %6;"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z),
        "l"(policy)
      : "memory");
}

// ------------------------------------------------------------------- tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {  // whole warp
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// D[tmem] (+)= A[smem] * B[smem]^T, e4m3 x e4m3 -> f32, one CTA; issued by ONE thread.
__device__ __forceinline__ void umma_f8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// mbarrier arrive once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// 32 lanes x 16 consecutive 32-bit columns -> 16 registers per thread (lane i of the
// warp reads TMEM lane (taddr.lane + i)); whole warp.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
// Waits for the loads above.  The wait names their registers, because the arithmetic on them is not volatile: without that
// nothing but the compiler's schedule would keep it behind the wait.
__device__ __forceinline__ void tmem_ld_wait_for(uint32_t (&r)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
               :: "memory");
}
__device__ __forceinline__ void tmem_ld_wait_for(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :: "memory");
}
__device__ __forceinline__ void tmem_ld_wait_for(uint32_t (&a)[16], uint32_t (&r)[16]) {
  tmem_ld_wait_for(a);
  asm volatile(""     // (no instruction: volatile statements keep their order)
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]));
}

// Packed pairs of f32 (sm_100 issues one FMA or multiply on both halves per instruction; each half is
// the IEEE operation, so results equal the scalar ones bit for bit).
__device__ __forceinline__ uint64_t f32x2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t f32x2_pack_bits(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void f32x2_unpack(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f32x2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t f32x2_mul(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Shared-memory matrix descriptor for a K-major operand tile stored as rows of 128
// bytes with the 128-byte swizzle (what a TMA load with SWIZZLE_128B writes): 8-row
// groups are 1024 bytes apart (stride byte offset), the leading byte offset is unused
// for swizzled K-major layouts (encoded 1), descriptor version 1, layout type 2.
// The tile base must be 1024-byte aligned; advancing K by 32 bytes inside the
// 128-byte row adds 2 to the (address >> 4) field.
__device__ __forceinline__ uint64_t umma_smem_desc_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(1) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}
// Instruction descriptor: f32 accumulator, A and B e4m3, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t umma_idesc_e4m3_m128(uint32_t n) {
  return (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// ------------------------------------------------------------------ CTA pairs
// Helpers for kernels launched as clusters of two CTAs whose tensor cores work on one tile
// (tcgen05 cta_group::2).  Addresses named "cluster address" are 32-bit shared::cluster
// addresses (mapa), which may point into the other CTA of the pair.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared-memory offset in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_u32(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
// every thread of both CTAs; orders everything before it (barrier inits included) cluster-wide
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void fence_acq_rel_cluster() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Arrive on a barrier in (possibly) the other CTA without a cluster-scope release: for hand-offs whose
// payload is tensor memory (ordered by tcgen05 fences), not ordinary memory.
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void st_cluster_f32(uint32_t cluster_addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(cluster_addr), "f"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t cluster_addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(cluster_addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster_u32(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
// Like mbar_wait_bounded, for barriers the other CTA of the pair arrives on (cluster-scope acquire);
// on expiry the failure code is also written into the other CTA's abort flag, so that its roles
// leave their loops at once instead of running into their own limits one after the other.
__device__ __forceinline__ bool mbar_wait_bounded_pair(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                       uint32_t peer_abort_cluster_addr, int code,
                                                       long long limit_cycles = (1ll << 31)) {
  if (mbar_try_wait_cluster(bar, parity)) return true;
  const long long t0 = clock64();
  while (true) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    if (*abort_flag != 0) return false;
    if (clock64() - t0 > limit_cycles) {
      *abort_flag = code;
      st_cluster_u32(peer_abort_cluster_addr, static_cast<uint32_t>(code));
      return false;
    }
  }
}
__device__ __forceinline__ bool mbar_try_wait_at(uint32_t bar, uint32_t parity) {
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
// The same for barriers that only this CTA's threads, its own loads or tcgen05.commit signal (CTA-scope
// acquire), still telling the partner when it gives up.  (Polling with mbarrier.test_wait instead of
// try_wait was measured and changed nothing.)  Shared-memory addresses, not pointers: the promotion warps have no
// registers to spare for 64-bit ones.
__device__ __forceinline__ bool mbar_wait_bounded_tell(uint32_t bar, uint32_t parity, uint32_t abort_flag, uint32_t peer_abort_cluster_addr,
                                                       int code, long long limit_cycles) {
  if (mbar_try_wait_at(bar, parity)) return true;
  const long long t0 = clock64();
  while (true) {
    if (mbar_try_wait_at(bar, parity)) return true;
    int aborted;
    asm volatile("ld.volatile.shared.s32 %0, [%1];" : "=r"(aborted) : "r"(abort_flag) : "memory");
    if (aborted != 0) return false;
    if (clock64() - t0 > limit_cycles) {
      asm volatile("st.volatile.shared.s32 [%0], %1;" ::"r"(abort_flag), "r"(code) : "memory");
      st_cluster_u32(peer_abort_cluster_addr, static_cast<uint32_t>(code));
      return false;
    }
  }
}
// as mbar_wait_or_clear
__device__ __forceinline__ void mbar_wait_or_clear_tell(bool& ok, uint32_t bar, uint32_t parity, uint32_t abort_flag,
                                                        uint32_t peer_abort_cluster_addr, int code, long long limit_cycles) {
  if (mbar_try_wait_at(bar, parity)) return;
  const long long t0 = clock64();
  while (ok && !mbar_try_wait_at(bar, parity)) {
    int aborted;
    asm volatile("ld.volatile.shared.s32 %0, [%1];" : "=r"(aborted) : "r"(abort_flag) : "memory");
    if (aborted != 0) {
      ok = false;
    } else if (clock64() - t0 > limit_cycles) {
      asm volatile("st.volatile.shared.s32 [%0], %1;" ::"r"(abort_flag), "r"(code) : "memory");
      st_cluster_u32(peer_abort_cluster_addr, static_cast<uint32_t>(code));
      ok = false;
    }
  }
}
// Tensor memory of both CTAs of the pair: the same warp of each CTA executes these.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// D (+)= A * B^T over the pair: M = 256 (each CTA's shared memory holds its 128 rows of A at the
// descriptor's offset, and its tensor memory receives the matching 128 rows of D), N columns of which
// each CTA's shared memory holds half the rows of B.  Issued by one thread of the pair's first CTA.
__device__ __forceinline__ void umma_f8_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the mbarrier at this shared-memory offset in every CTA of `cta_mask` once the pair's MMAs
// issued so far have completed (a signal only: no data is copied between CTAs).
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar, uint16_t cta_mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"(cta_mask)
               : "memory");
}
__host__ __device__ constexpr uint32_t umma_idesc_e4m3_m256(uint32_t n) {
  return (1u << 4) | ((n >> 3) << 17) | ((256u >> 4) << 24);
}
// Tiled load into THIS CTA's shared memory whose completion is counted on an mbarrier that may live in
// the other CTA of the pair (cluster address).  One CTA's data only: nothing is multicast.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* m, uint32_t bar_cluster_addr,
                                                 int x, int y, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster_addr), "r"(x), "r"(y),
        "l"(policy)
      : "memory");
}

// ------------------------------------------------------------- cp.async (4 B)
// Untiled bulk copy global -> shared (both addresses 16-byte aligned, size a multiple of 16 bytes),
// completion counted in bytes on an mbarrier like the tiled loads.
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gmem_src, uint32_t bytes, uint64_t* bar,
                                          uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
      :: "r"(smem_u32(smem_dst)), "l"(gmem_src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}

// ------------------------------------------------------------ small helpers
// 16-byte load through the coherent path (not ld.global.nc): for data another kernel that may still be
// running has written and released
__device__ __forceinline__ float4 ld_global_f32x4(const float* p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
// 4x4 transposes across a lane quad (lanes 4q..4q+3).  Before: lane r holds row r = (m[r][0..3]).
// After: lane c holds column c = (m[0..3][c]).  Used to turn "one feature, four token rows" per
// thread into "four adjacent features of one token row", so a store carries 4x the bytes.
__device__ __forceinline__ uint32_t quad_transpose_bytes(uint32_t v, int lane) {
  const uint32_t o1 = __shfl_xor_sync(0xffffffffu, v, 1);
  v = (lane & 1) ? __byte_perm(v, o1, 0x3715) : __byte_perm(v, o1, 0x6240);
  const uint32_t o2 = __shfl_xor_sync(0xffffffffu, v, 2);
  return (lane & 2) ? __byte_perm(v, o2, 0x3276) : __byte_perm(v, o2, 0x5410);
}
__device__ __forceinline__ void quad_transpose_f32(float& a0, float& a1, float& a2, float& a3, int lane) {
  {
    const bool odd = lane & 1;
    const float rx = __shfl_xor_sync(0xffffffffu, odd ? a0 : a1, 1);
    const float ry = __shfl_xor_sync(0xffffffffu, odd ? a2 : a3, 1);
    if (odd) { a0 = rx; a2 = ry; } else { a1 = rx; a3 = ry; }
  }
  {
    const bool hi = lane & 2;
    const float rx = __shfl_xor_sync(0xffffffffu, hi ? a0 : a2, 2);
    const float ry = __shfl_xor_sync(0xffffffffu, hi ? a1 : a3, 2);
    if (hi) { a0 = rx; a1 = ry; } else { a2 = rx; a3 = ry; }
  }
}

// two floats -> two e4m3 bytes (lo -> bits 0..7, hi -> bits 8..15), round-nearest, saturating
__device__ __forceinline__ uint16_t cvt_e4m3x2(float lo, float hi) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float2 e4m3x2_to_float2(uint16_t v) {
  uint32_t h2;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(v));
  __half2 h = *reinterpret_cast<__half2*>(&h2);
  return __half22float2(h);
}

}  // namespace syfi

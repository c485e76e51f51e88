// mbarrier helpers: bounded waits on bytes that copies or other CTAs of a
// cluster deliver.
#pragma once

#include "pmg_common.cuh"

namespace pmg {

// mbarrier polls before the stage counts as lost: about 0.1 s, some 10^4
// times the longest real wait
constexpr long kTmaMaxPolls = 1L << 20;

__device__ __forceinline__ unsigned smem_addr(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(
                   smem_addr(bar)),
               "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar,
                                               unsigned bytes) {
  asm volatile(
      "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(
          smem_addr(bar)),
      "r"(bytes)
      : "memory");
}
// true once the phase with this parity has completed
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar,
                                              unsigned parity) {
  unsigned done;
  asm volatile("{\n"
               ".reg .pred p;\n"
               "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
               "selp.u32 %0, 1, 0, p;\n"
               "}\n"
               : "=r"(done)
               : "r"(smem_addr(bar)), "r"(parity)
               : "memory");
  return done != 0;
}
// bounded wait: false if the phase did not complete within kTmaMaxPolls
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity) {
  for (long n = 0; n < kTmaMaxPolls; ++n) {
    if (mbar_try_wait(bar, parity))
      return true;
    if (n > 64)
      __nanosleep(64);
  }
  return false;
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}

// ---- messages between the CTAs of a cluster ---------------------------------
// A value stored into another CTA's shared memory together with its bytes on
// that CTA's mbarrier: the receiver waits for the bytes it expects, where a
// cluster barrier would wait for every CTA and every store (the two sums of
// a CG iteration, cg_cluster.cuh: 2.1 -> 1.5 us at 11^3).

// the address of this CTA's shared object in CTA `rank` of the cluster
__device__ __forceinline__ unsigned cluster_addr(const void *p, int rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;\n"
      : "=r"(r)
      : "r"(smem_addr(p)), "r"(rank));
  return r;
}
// Nothing is sent where bar is 0. The test is a predicate, not a branch: a
// branch that only some lanes take, around an asm statement, leaves the warp
// split for the rest of the kernel (every later shuffle and warp barrier
// slower, measured 120 against 15 ns).
__device__ __forceinline__ void send(unsigned dst, double v, unsigned bar) {
  asm volatile("{\n"
               ".reg .pred p;\n"
               "setp.ne.u32 p, %2, 0;\n"
               "@p st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 "
               "[%0], %1, [%2];\n"
               "}\n" ::"r"(dst),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void send(unsigned dst, float v, unsigned bar) {
  asm volatile("{\n"
               ".reg .pred p;\n"
               "setp.ne.u32 p, %2, 0;\n"
               "@p st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 "
               "[%0], %1, [%2];\n"
               "}\n" ::"r"(dst),
               "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}
// mbar_expect_tx in the threads with `on`
__device__ __forceinline__ void mbar_expect_tx_if(bool on, uint64_t *bar,
                                                  unsigned bytes) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.u32 p, %2, 0;\n"
      "@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n"
      "}\n" ::"r"(smem_addr(bar)),
      "r"(bytes), "r"((unsigned)on)
      : "memory");
}
// In the threads with `on`: `bytes` (a multiple of 16) of this CTA's shared
// memory, written and fenced (fence_proxy_async_smem), to the 16-byte aligned
// cluster address dst, completing on that CTA's mbarrier.
__device__ __forceinline__ void copy_to_cta_if(bool on, unsigned dst,
                                               const void *src,
                                               unsigned bytes, unsigned bar) {
  asm volatile("{\n"
               ".reg .pred p;\n"
               "setp.ne.u32 p, %4, 0;\n"
               "@p cp.async.bulk.shared::cluster.shared::cta.mbarrier::"
               "complete_tx::bytes [%0], [%1], %2, [%3];\n"
               "}\n" ::"r"(dst),
               "r"(smem_addr(src)), "r"(bytes), "r"(bar), "r"((unsigned)on)
               : "memory");
}
// Polls for a message before it counts as lost: the hardware suspends a poll
// that finds nothing for about 4 us, so a quarter of a second, ten times the
// longest wait there is (a CTA waiting out 20000 iterations of the level-1 CG
// in another).
constexpr int kMessagePolls = 1 << 16;

// mbar_wait for messages: what the senders wrote before them is visible. A
// thread that has lost a message before looks once and goes on.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t *bar,
                                                  unsigned parity,
                                                  bool lost) {
  const int limit = lost ? 1 : kMessagePolls;
  for (int polls = 0; polls < limit; ++polls) {
    unsigned done;
    asm volatile("{\n"
                 ".reg .pred p;\n"
                 "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 "
                 "p, [%1], %2;\n"
                 "selp.u32 %0, 1, 0, p;\n"
                 "}\n"
                 : "=r"(done)
                 : "r"(smem_addr(bar)), "r"(parity)
                 : "memory");
    if (done)
      return true;
  }
  return false;
}

// The end of a kernel whose CTAs send to each other: no CTA leaves while
// another may still send to it. A CTA that has received everything it expects
// can leave after the barrier; one with a thread that lost a message stays
// another millisecond (some 10^3 times a message), so that what was sent to
// it before the barrier lands in its own memory.
__device__ __forceinline__ void leave_cluster(bool lost) {
  asm volatile("barrier.cluster.arrive;\n"
               "barrier.cluster.wait;\n" ::
                   : "memory");
  if (lost)
    for (int q = 0; q < 64; ++q)
      __nanosleep(16384);
}

} // namespace pmg

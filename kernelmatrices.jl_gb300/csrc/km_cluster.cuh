// Stores and waits between the CTAs of a thread-block cluster: addresses in another CTA's shared
// memory, asynchronous stores that complete a barrier there, bounded waits on a barrier.
#pragma once

#include <cuda_runtime.h>

namespace km {

// Polls before a wait on a barrier or a shared-memory flag gives up: a few tens of cycles each, so well
// above any legitimate wait inside one leaf or node, far below a watchdog.  (Not a time: the clock also
// runs while the process has been switched off the GPU for another one.)
constexpr int kWaitPolls = 1 << 22;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// the address of shared-memory location `a` in CTA `rank` of the cluster
__device__ __forceinline__ unsigned at_rank(unsigned a, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}

// 8 bytes to another CTA's shared memory; they count towards that CTA's barrier
__device__ __forceinline__ void st_async(unsigned addr, double v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}

// n bytes (a multiple of 16, both addresses too) of this CTA's shared memory to another's; they count
// towards that CTA's barrier.  Stores by this CTA's threads come before a fence.proxy.async.
__device__ __forceinline__ void copy_to_rank(unsigned dst, unsigned src, unsigned n, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "r"(src), "r"(n), "r"(bar)
               : "memory");
}

// Cluster instructions (mapa, st.async, cluster-scope waits) are for launches with a cluster
// dimension only: in a plain launch the node kernel's st.async raised an illegal instruction.  A
// one-CTA node therefore stores locally and arrives on the barrier itself.
__device__ __forceinline__ bool bar_try(unsigned bar, int cs) {
  unsigned ok;
  if (cs > 1)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar)
        : "memory");
  return ok != 0;
}

// Waits for phase 0 of the barrier; false if it gave up (after wait_limit polls, < 0: kWaitPolls)
__device__ __forceinline__ bool bar_wait(unsigned bar, int wait_limit, int cs) {
  const int lim = wait_limit < 0 ? kWaitPolls : wait_limit;
  int n = 0;
  while (wait_limit == 0 || !bar_try(bar, cs))
    if (++n > lim) return false;
  return true;
}

}  // namespace km

// mbarrier and bulk-copy helpers of the dedispersion kernels.
#pragma once
#include <cuda_runtime.h>

namespace vfrb {

// mbarrier and bulk-copy helpers (sm_90+ PTX; no multicast)
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
// Waits for the barrier phase with the given parity; gives up (false) after
// a bounded number of polls instead of spinning for ever.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) {
  const unsigned a = smem_u32(bar);
  for (int i = 0; i < (1 << 22); ++i) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
// bytes from global to this CTA's shared memory, completing on `bar` (16-byte
// aligned addresses, size a multiple of 16)
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// A warp whose wait for chunk k (buffer k & 1) gave up stages nothing more; its copies
// of that chunk and of the next one, which it has staged, must land before its CTA's
// shared memory is used otherwise.  (It may not arrive for another chunk, whose phase
// could run into this one; the others' waits then give up as well.)  Bounded too.  Out
// of line: inside the loop it cost the kernel registers (201 trials 583 us, 579).
static __device__ __noinline__ void drain_copies(unsigned long long* full, int k, int nchunks) {
  mbar_wait(&full[k & 1], (unsigned)(k >> 1) & 1u);
  if (k + 1 < nchunks) mbar_wait(&full[(k + 1) & 1], (unsigned)((k + 1) >> 1) & 1u);
}

}  // namespace vfrb

// Asynchronous bulk copies global -> shared memory with mbarrier completion
// (sm_90 and later, here sm_103a), written as inline PTX.
//
// A stage buffer is filled by one thread: it arms the stage's mbarrier with
// the byte count it expects (arrive.expect_tx) and issues cp.async.bulk
// copies that complete bytes on that barrier.  Consumers wait on the phase
// parity of the barrier.  Every wait is bounded in time: a wait that runs
// out returns false, and the caller records the failure in the handle's
// status word instead of spinning forever.
#pragma once
#include <cstdint>

namespace hcd {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

// makes the initialised barriers visible to the asynchronous proxy
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// Waits for the phase of `parity` to complete; gives up after `limit` clock
// cycles (about a second at the SM clock when limit = 2e9).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, long long limit) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity))
    if (clock64() - t0 > limit) return false;
  return true;
}

// One contiguous global -> shared copy; dst, src and bytes are multiples of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// Programmatic dependent launch (sm_90 and later).  A kernel launched with
// the programmatic-serialisation attribute may start while the kernel before
// it in the stream is still draining; it must wait (pdl_wait) before it
// reads anything that kernel writes.  pdl_trigger marks the calling CTA's
// share of the work as issued, so that the next kernel can be launched once
// every CTA has triggered or exited.  Both are no-ops for a kernel launched
// without the attribute.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Thread-block clusters: the CTA's rank and the cluster's size, a barrier over
// every thread of the cluster (release on arrival, acquire on the wait, so that
// global and shared writes before it are seen after it), and loads from the
// shared memory of another CTA of the cluster at the address `a` has there.
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// A cluster of one needs no more than the CTA's barrier (the cluster's costs a
// memory barrier and a cold L1 on top).
__device__ __forceinline__ void cluster_sync(int size) {
  if (size > 1) {
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ int ld_cluster_int(uint32_t a) {
  int v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void ld_cluster(uint32_t a, float& v) {
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
}
__device__ __forceinline__ void ld_cluster(uint32_t a, double& v) {
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
}
// the same from the CTA's own shared memory
__device__ __forceinline__ void ld_shared(uint32_t a, float& v) {
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
}
__device__ __forceinline__ void ld_shared(uint32_t a, double& v) {
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
}
__device__ __forceinline__ void ld_shared4(uint32_t a, float* v) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(a));
}
__device__ __forceinline__ void ld_shared4(uint32_t a, double* v) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(a));
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[2]), "=d"(v[3]) : "r"(a + 16));
}
// four values from a 16-byte aligned address
__device__ __forceinline__ void ld_cluster4(uint32_t a, float* v) {
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(a));
}
__device__ __forceinline__ void ld_cluster4(uint32_t a, double* v) {
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(a));
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v[2]), "=d"(v[3]) : "r"(a + 16));
}

}  // namespace hcd

// fgpu_bulk.cuh -- PTX wrappers of the asynchronous copies that stage planes and rows in shared
// memory: mbarriers, bulk tensor copies, 8-byte cp.async, L2 prefetches.
#pragma once
#include <cuda.h>
#include "fgpu_device.cuh"

namespace fgpu {

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
// orders this thread's generic-proxy shared-memory accesses with later async-proxy ones
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_test(unsigned long long* b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Wait for phase `parity` of an mbarrier, for at most about two seconds of SM clock;
// false when the limit ran out.
__device__ __forceinline__ bool mbar_wait(unsigned long long* b, unsigned parity) {
  if (mbar_test(b, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_test(b, parity))
    if (clock64() - t0 > 4000000000LL) return false;
  return true;
}
// bulk tensor copy of one box (coordinates x, y, z; the variable coordinate 0) into shared
// memory, completing on the mbarrier; RANK 4 (x, y, z, var) or 3 (x, y, var)
template <int RANK>
__device__ __forceinline__ void tma_load_box(void* dst, const CUtensorMap* map, unsigned long long* bar, int x, int y,
                                             int z) {
  if (RANK == 4)
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];" ::"r"(smem_addr(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(0), "r"(smem_addr(bar))
        : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(smem_addr(dst)),
        "l"(map), "r"(x), "r"(y), "r"(0), "r"(smem_addr(bar))
        : "memory");
}
// L2 prefetch of `bytes` contiguous bytes (16-byte aligned address, multiple of 16 bytes)
__device__ __forceinline__ void bulk_prefetch_l2(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// asynchronous copy of one double; completion is counted by cp_async_arrive
__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
// one arrival on the mbarrier once this thread's copies so far have landed
__device__ __forceinline__ void cp_async_arrive(unsigned long long* b) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The interior index whose raw value is fetched for index x of an axis of n cells: periodic faces
// (bc[0] low, bc[1] high) wrap, others clamp (their ghosts are computed from interior values).
__device__ __forceinline__ int wrap_index(int x, int n, const int* bc) {
  if (x < 0 && bc[0] == BC_PERIODIC) x += n;
  else if (x >= n && bc[1] == BC_PERIODIC) x -= n;
  return min(max(x, 0), n - 1);
}

}  // namespace fgpu

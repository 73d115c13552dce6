// Helpers of the pipelined, warp-specialised M-update kernels (k_mupdate2.cu for num_wann <= 32,
// k_mupdate3.cu for 33..128): the stage layout, named and memory barriers, bounded waits.
#pragma once
#include "oz.cuh"

namespace w90g {

namespace {

constexpr int kDynBudget = 232448 - 5120;                 // opt-in smem minus static use and slack

// element (r, q) of a 128 x 16 K-major stage plane (canonical layout, no swizzle):
// core matrices of 8 rows x 8 K (16 B rows), LBO 128 B along K, SBO 256 B along rows
__device__ __forceinline__ uint32_t stage_off(int r, int q) {
  return (uint32_t)((r >> 3) * 256 + (q >> 3) * 128 + (r & 7) * 16 + (q & 7) * 2);
}

__device__ __forceinline__ void bar_named(int id, int n) {
  asm volatile("bar.sync %0, %1;" :: "r"(id), "r"(n) : "memory");
}

// bounded wait that also stops when another role reported a failure (*bad != 0)
__device__ __forceinline__ bool mbar_wait_role(uint32_t addr, uint32_t parity, volatile int* bad) {
  for (int it = 0; it < W90G_SPIN_LIMIT; ++it) {
    if (mbar_try(addr, parity)) return true;
    if ((it & 63) == 63 && *bad) return false;
  }
  return false;
}

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(b)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" :: "r"(smem_u32(b)) : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* b) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
               :: "r"(smem_u32(b)) : "memory");
}

// the group's skip predicate, read alike by every role (nothing writes it during the kernel)
__device__ __forceinline__ bool group_active(const Problem& P, int which) {
  const CtrlState* st = P.st;
  return !st->done && !(which == 1 && !st->do_second);
}

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) !=
                                                  cudaSuccess || n <= 0)
      n = 148;
  }
  return n;
}

}  // namespace

}  // namespace w90g

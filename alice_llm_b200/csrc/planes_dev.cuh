// What the kernels over ternary planes and packed codes share (csrc/gemv_planes.cu, csrc/gemv_planes_tc.cu).
#pragma once
#include "digits_dev.cuh"

namespace alice {

__device__ __forceinline__ bool can_vec4(const float* x, uint32_t cols) { return cols % 4 == 0 && ((uintptr_t)x & 15) == 0; }
__device__ __forceinline__ long long ld_cluster_s64(uint32_t addr, uint32_t rank) {
    uint32_t remote;
    long long v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.s64 %0, [%1];" : "=l"(v) : "r"(remote) : "memory");
    return v;
}

}  // namespace alice

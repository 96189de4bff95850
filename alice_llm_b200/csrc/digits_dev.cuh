// Largest magnitude of an f32 vector by a whole CTA, for the fixed-point digits of csrc/gemv_planes.cu and csrc/gemv_blocks.cu.
#pragma once
#include "common.cuh"

namespace alice {

// THREADS threads take part; red = THREADS / 32 floats of shared memory. 16 loads of 16 bytes a thread are in flight at once.
template <int THREADS>
static __device__ __forceinline__ float vec_amax(const float* x, uint32_t n, bool vec4, float* red, bool& finite) {
    const uint32_t tid = threadIdx.x;
    float amax = 0.0f, odd = 0.0f;         // odd: stays 0 for a finite vector (inf * 0 and NaN * 0 are NaN)
    if (vec4) {
        for (uint32_t base = 0; base < n / 4; base += THREADS * 16) {
            float4 q[16];
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const uint32_t i = base + k * THREADS + tid;
                q[k] = i < n / 4 ? __ldcg(reinterpret_cast<const float4*>(x) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int k = 0; k < 16; k++) {
                amax = fmaxf(fmaxf(amax, fmaxf(fabsf(q[k].x), fabsf(q[k].y))), fmaxf(fabsf(q[k].z), fabsf(q[k].w)));
                odd = fmaf(q[k].x, 0.0f, fmaf(q[k].y, 0.0f, fmaf(q[k].z, 0.0f, fmaf(q[k].w, 0.0f, odd))));
            }
        }
    } else {
        for (uint32_t i = tid; i < n; i += THREADS) {
            const float q = __ldcg(x + i);
            amax = fmaxf(amax, fabsf(q));
            odd = fmaf(q, 0.0f, odd);
        }
    }
    finite = __syncthreads_and(odd == 0.0f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if ((tid & 31) == 0) red[tid >> 5] = amax;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < THREADS / 32; w++) amax = fmaxf(amax, red[w]);
    return amax;
}

}  // namespace alice

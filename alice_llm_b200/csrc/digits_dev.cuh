// Fixed point of f32 vectors, for the digits of csrc/gemv_mma.cuh, csrc/gemv_planes.cu and csrc/gemv_blocks.cu: its unit, and the largest
// magnitude of a vector by a whole CTA.
#pragma once
#include "common.cuh"

namespace alice {

// A factor 2^n, n up to 149, that takes f32 numbers to units: two factors, since 2^128 is no f32.
struct FixedScale { float a, b; };
__device__ __forceinline__ int to_units(float x, const FixedScale& s) { return __float2int_rn(x * s.a * s.b); }
// A unit is BITS bits below a power of two above amax, but not below 2^-149, of which every f32 number is a whole multiple. kappa: its
// value. A vector that is not finite has units of NaN, and so have all its results.
template <int BITS>
__device__ __forceinline__ void fixed_scale(float amax, bool finite, FixedScale& to_fixed, float& kappa) {
    const uint32_t ebits = (__float_as_uint(amax) >> 23) & 0xffu;
    const int n = ebits == 0xffu ? BITS : min(BITS + 126 - (int)ebits, 149);
    to_fixed = {finite ? ldexpf(1.0f, min(n, 100)) : 0.0f, ldexpf(1.0f, max(n - 100, 0))};
    kappa = finite ? ldexpf(1.0f, -n) : __int_as_float(0x7fffffff);
}

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

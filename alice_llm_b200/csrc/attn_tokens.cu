// Attention of several consecutive tokens of a Llama-style model, everything in f32: a verify step or a piece of a prompt.
// Arithmetic as csrc/attn_body.cuh (apply_rope src/llama3.rs:5323-5333, KvCache::append :4773, gqa_attention :5431-5690), causal
// by src/shaders/attention.wgsl:45.
//
// Token by token (the decode kernel with one CTA per token) every token reads the whole context again and every score is a
// shuffle reduction: 131 us a layer for eight tokens of a 64-head model behind 2048. Here the tokens x query heads of one key /
// value head are the rows of a tile, as in a matrix product: 64 rows x 32 keys per step, K and V brought in once per tile
// with cp.async while the step before computes, scores and weighted sums from 4 x 2 and 4 x 8 register blocks: 38 us for the same
// layer (tiles 24.5, join 10, append 3.6). What bounds it: the f32 pipe, and shared-memory reads within 20 % of it.
#include <algorithm>
#include <type_traits>

#include "attn_body.cuh"
#include "common.cuh"
#include "glue.cuh"

namespace alice {
namespace {

constexpr int AT_ROWS = 64, AT_KEYS = 32, AT_PITCH = 132;   // pitch in floats: rows 16 bytes apart modulo 128, so 8 rows fill the banks
constexpr uint32_t AT_TILE = AT_KEYS * AT_PITCH;
constexpr uint32_t AT_SMEM = (AT_ROWS * AT_PITCH + 4 * AT_TILE + AT_ROWS * (AT_KEYS + 4)) * 4;

__device__ __forceinline__ float4 lds4f(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}

// Rotates the queries in place and appends the rotated keys and the values to the cache: a warp per head vector.
__global__ void __launch_bounds__(256) attn_append_kernel(const __grid_constant__ AttnArgs a, float* qkv, uint32_t batch) {
    pdl_launch_dependents();
    pdl_wait();
    const AttnShape s = a.shape;
    const uint32_t lane = threadIdx.x & 31, hv = s.num_heads + 2 * s.num_kv_heads;
    const uint32_t i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= hv * batch) return;
    const uint32_t k = i / hv, h = i % hv, kv_dim = s.num_kv_heads * 128;
    float4* src = reinterpret_cast<float4*>(qkv + (size_t)k * hv * 128 + (size_t)h * 128) + lane;
    float4 v = __ldcg(src);
    const size_t t = (size_t)(uint32_t)*a.pos + k;
    if (h < s.num_heads + s.num_kv_heads) v = rope4(v, lane, rope_coef(a.rope_tab + (size_t)k * 128, lane, a.neox), a.neox);
    if (h < s.num_heads) *src = v;
    else if (h < s.num_heads + s.num_kv_heads) reinterpret_cast<float4*>(a.kcache + t * kv_dim + (size_t)(h - s.num_heads) * 128)[lane] = v;
    else reinterpret_cast<float4*>(a.vcache + t * kv_dim + (size_t)(h - s.num_heads - s.num_kv_heads) * 128)[lane] = v;
}

// blockIdx: key / value head, tile of 64 (token, head) rows, share of the positions. nsplit == 1: the finished output; else
// (max, sum, sums) of the share into a.part[row][split].
template <int GROUP>
__global__ void __launch_bounds__(256, 2) attn_tile_kernel(const __grid_constant__ AttnArgs a, uint32_t batch) {
    extern __shared__ __align__(16) float sm[];
    float* sq = sm;
    float* sk = sq + AT_ROWS * AT_PITCH;             // [2][keys]
    float* sv = sk + 2 * AT_TILE;
    float* sp = sv + 2 * AT_TILE;                    // [rows][keys + 4]
    const AttnShape s = a.shape;
    const uint32_t kvh = blockIdx.x, row0 = blockIdx.y * AT_ROWS, split = blockIdx.z;
    const uint32_t tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, kv_dim = s.num_kv_heads * 128;
    const uint32_t qkv_stride = (s.num_heads + 2 * s.num_kv_heads) * 128, nrows = batch * GROUP;
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t pos0 = (uint32_t)*a.pos;
    const uint32_t seen = pos0 + min(batch, (row0 + AT_ROWS - 1) / GROUP + 1);   // positions the last row of the tile sees
    const uint32_t per = ((pos0 + batch + a.nsplit - 1) / a.nsplit + AT_KEYS - 1) / AT_KEYS * AT_KEYS;
    const uint32_t t0 = split * per, t1 = min(seen, t0 + per);
    const uint32_t steps = t1 > t0 ? (t1 - t0 + AT_KEYS - 1) / AT_KEYS : 0u;

    auto fetch = [&](uint32_t step) {
        const uint32_t tb = t0 + step * AT_KEYS, b = (step & 1) * AT_TILE;
#pragma unroll
        for (uint32_t i = tid; i < AT_KEYS * 32; i += 256) {
            const uint32_t r = i >> 5, c = (i & 31) * 4, t = min(tb + r, t1 - 1);     // keys past the share are masked
            const size_t at = (size_t)t * kv_dim + kvh * 128 + c;
            cp16(smem_u32(sk + b + r * AT_PITCH + c), a.kcache + at);
            cp16(smem_u32(sv + b + r * AT_PITCH + c), a.vcache + at);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (uint32_t i = tid; i < AT_ROWS * 32; i += 256) {
        const uint32_t r = i >> 5, c = (i & 31) * 4, row = min(row0 + r, nrows - 1);
        cp16(smem_u32(sq + r * AT_PITCH + c), a.qkv + (size_t)(row / GROUP) * qkv_stride + (kvh * GROUP + row % GROUP) * 128 + c);
    }
    if (steps) fetch(0); else asm volatile("cp.async.commit_group;" ::: "memory");

    const float inv_sqrt_d = __fdiv_rn(1.0f, sqrtf(128.0f));
    float m[4], l[4], o[4][8];
    uint32_t last[4];                               // first position the row does not see
    const uint32_t all_see = min(t1, pos0 + row0 / GROUP + 1);      // positions below it are seen by every row of the tile
#pragma unroll
    for (int i = 0; i < 4; i++) {
        m[i] = -INFINITY; l[i] = 0.0f;
        last[i] = min(t1, pos0 + (row0 + ty * 4 + i) / GROUP + 1);
#pragma unroll
        for (int d = 0; d < 8; d++) o[i][d] = 0.0f;
    }
    for (uint32_t step = 0; step < steps; step++) {
        if (step + 1 < steps) fetch(step + 1);
        if (step + 1 < steps) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const uint32_t b = (step & 1) * AT_TILE, tb = t0 + step * AT_KEYS;
        const uint32_t qa = smem_u32(sq + ty * 4 * AT_PITCH), ka = smem_u32(sk + b + tx * AT_PITCH);
        float sc[4][2] = {};
#pragma unroll 4
        for (uint32_t c = 0; c < 32; c++) {
            const float4 k0 = lds4f(ka + c * 16), k1 = lds4f(ka + 16 * AT_PITCH * 4 + c * 16);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 q = lds4f(qa + i * AT_PITCH * 4 + c * 16);
                sc[i][0] = fmaf(q.x, k0.x, fmaf(q.y, k0.y, fmaf(q.z, k0.z, fmaf(q.w, k0.w, sc[i][0]))));
                sc[i][1] = fmaf(q.x, k1.x, fmaf(q.y, k1.y, fmaf(q.z, k1.z, fmaf(q.w, k1.w, sc[i][1]))));
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 2; j++) {
                sc[i][j] = tb + tx + 16 * j < last[i] ? sc[i][j] * inv_sqrt_d : -INFINITY;
                mx = fmaxf(mx, sc[i][j]);
            }
#pragma unroll
            for (int w = 8; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
            const float mn = fmaxf(m[i], mx);
            const float corr = m[i] == mn ? 1.0f : expf(m[i] - mn);        // a row that has seen nothing: -inf == -inf
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const float p = sc[i][j] == -INFINITY ? 0.0f : expf(sc[i][j] - mn);
                sp[(ty * 4 + i) * (AT_KEYS + 4) + tx + 16 * j] = p;
                sum += p;
            }
#pragma unroll
            for (int w = 8; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
            l[i] = l[i] * corr + sum;
            m[i] = mn;
#pragma unroll
            for (int d = 0; d < 8; d++) o[i][d] *= corr;
        }
        __syncwarp();      // the 16 threads of a row are half a warp
        const uint32_t pa = smem_u32(sp + ty * 4 * (AT_KEYS + 4)), va = smem_u32(sv + b + tx * 4);
        auto weigh = [&](auto masked) {
#pragma unroll 2
            for (uint32_t t = 0; t < AT_KEYS; t += 4) {
                float4 p[4];
#pragma unroll
                for (int i = 0; i < 4; i++) p[i] = lds4f(pa + i * (AT_KEYS + 4) * 4 + t * 4);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float4 v0 = lds4f(va + (t + j) * AT_PITCH * 4), v1 = lds4f(va + (t + j) * AT_PITCH * 4 + 256);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (masked.value && tb + t + j >= last[i]) continue;      // a value the row does not see may be infinite: 0 times it is not 0
                        const float w = j == 0 ? p[i].x : j == 1 ? p[i].y : j == 2 ? p[i].z : p[i].w;
                        o[i][0] = fmaf(w, v0.x, o[i][0]); o[i][1] = fmaf(w, v0.y, o[i][1]); o[i][2] = fmaf(w, v0.z, o[i][2]); o[i][3] = fmaf(w, v0.w, o[i][3]);
                        o[i][4] = fmaf(w, v1.x, o[i][4]); o[i][5] = fmaf(w, v1.y, o[i][5]); o[i][6] = fmaf(w, v1.z, o[i][6]); o[i][7] = fmaf(w, v1.w, o[i][7]);
                    }
                }
            }
        };
        if (tb + AT_KEYS <= all_see) weigh(std::false_type{}); else weigh(std::true_type{});
        __syncthreads();   // this half of the K and V tiles is free
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t row = row0 + ty * 4 + i;
        if (row >= nrows) continue;
        const uint32_t k = row / GROUP, head = kvh * GROUP + row % GROUP;
        float* out;
        float f = 1.0f;
        if (a.nsplit == 1) {
            out = a.attn_out + (size_t)k * a.out_stride + (size_t)head * 128;
            f = l[i] > 0.0f ? 1.0f / l[i] : 0.0f;
        } else {
            out = a.part + (((size_t)k * s.num_heads + head) * a.nsplit + split) * 132;
            if (tx == 0) { out[0] = m[i]; out[1] = l[i]; }
            out += 4;
        }
        reinterpret_cast<float4*>(out)[tx] = make_float4(o[i][0] * f, o[i][1] * f, o[i][2] * f, o[i][3] * f);
        reinterpret_cast<float4*>(out)[16 + tx] = make_float4(o[i][4] * f, o[i][5] * f, o[i][6] * f, o[i][7] * f);
    }
}

// Joins the shares of one (token, head): a warp each, four dimensions a lane.
__global__ void __launch_bounds__(256) attn_join_kernel(const __grid_constant__ AttnArgs a, uint32_t vectors) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= vectors) return;
    const float* part = a.part + (size_t)i * a.nsplit * 132;
    float M = -INFINITY;
    for (uint32_t sp = lane; sp < a.nsplit; sp += 32) M = fmaxf(M, __ldcg(part + sp * 132));
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, w));
    float L = 0.0f;
    float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t sp0 = 0; sp0 < a.nsplit; sp0 += 8) {
        float2 ml[8];
        float4 v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float* p = part + min(sp0 + j, a.nsplit - 1) * 132;
            ml[j] = __ldcg(reinterpret_cast<const float2*>(p));
            v[j] = __ldcg(reinterpret_cast<const float4*>(p + 4) + lane);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (sp0 + j < a.nsplit) {      // a share without a maximum: nothing seen (all zeros), or nothing but NaN, which stays
                const float c = ml[j].x == -INFINITY ? 0.0f : expf(ml[j].x - M);
                L += ml[j].y * c;
                A.x += v[j].x * c; A.y += v[j].y * c; A.z += v[j].z * c; A.w += v[j].w * c;
            }
        }
    }
    const float inv = L > 0.0f ? 1.0f / L : 0.0f;
    const uint32_t k = i / a.shape.num_heads, head = i % a.shape.num_heads;
    reinterpret_cast<float4*>(a.attn_out + (size_t)k * a.out_stride + (size_t)head * 128)[lane] = make_float4(A.x * inv, A.y * inv, A.z * inv, A.w * inv);
}

template <int GROUP>
cudaError_t launch_tile(cudaLaunchConfig_t& lc, const AttnArgs& a, uint32_t batch) {
    static bool done[64] = {};
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev >= 64 || !done[dev]) {
        err = cudaFuncSetAttribute(attn_tile_kernel<GROUP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AT_SMEM);
        if (err != cudaSuccess) return err;
        if (dev < 64) done[dev] = true;
    }
    lc.dynamicSmemBytes = AT_SMEM;
    return cudaLaunchKernelEx(&lc, attn_tile_kernel<GROUP>, a, batch);
}

}  // namespace

cudaError_t launch_attention_tokens(const AttnArgs& args, float* qkv, uint32_t batch, uint32_t pos0, uint32_t part_vectors, int num_sms, cudaStream_t st, bool pdl) {
    AttnArgs a = args;
    const AttnShape& s = a.shape;
    if (s.head_dim != 128 || s.num_heads % s.num_kv_heads || a.npeers) return cudaErrorInvalidValue;
    const uint32_t group = s.num_heads / s.num_kv_heads, tiles = (batch * group + AT_ROWS - 1) / AT_ROWS;
    // shares of the positions: two CTAs an SM, at least two steps each, as many as the scratch holds
    const uint32_t want = (2 * (uint32_t)num_sms) / (s.num_kv_heads * tiles), most = (pos0 + batch + 2 * AT_KEYS - 1) / (2 * AT_KEYS);
    a.nsplit = std::max<uint32_t>(1, std::min({want, most, part_vectors / (batch * s.num_heads)}));
    cudaLaunchConfig_t lc = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at; lc.numAttrs = pdl ? 1 : 0; lc.stream = st; lc.blockDim = dim3(256);
    lc.gridDim = dim3(((s.num_heads + 2 * s.num_kv_heads) * batch + 7) / 8);
    cudaError_t err = cudaLaunchKernelEx(&lc, attn_append_kernel, a, qkv, batch);
    if (err != cudaSuccess) return err;
    lc.gridDim = dim3(s.num_kv_heads, tiles, a.nsplit);
    switch (group) {
        case 1: err = launch_tile<1>(lc, a, batch); break;
        case 2: err = launch_tile<2>(lc, a, batch); break;
        case 4: err = launch_tile<4>(lc, a, batch); break;
        case 5: err = launch_tile<5>(lc, a, batch); break;
        case 8: err = launch_tile<8>(lc, a, batch); break;
        default: err = cudaErrorInvalidValue;
    }
    if (err != cudaSuccess || a.nsplit == 1) return err;
    lc.gridDim = dim3((batch * s.num_heads + 7) / 8); lc.dynamicSmemBytes = 0;
    return cudaLaunchKernelEx(&lc, attn_join_kernel, a, batch * s.num_heads);
}

}  // namespace alice

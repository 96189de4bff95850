// Attention of several consecutive tokens of a Llama-style model, everything in f32: a verify step or a piece of a prompt.
// Arithmetic as csrc/attn_body.cuh (apply_rope src/llama3.rs:5323-5333, KvCache::append :4773, gqa_attention :5431-5690), causal
// by src/shaders/attention.wgsl:45.
//
// Token by token (the decode kernel with one CTA per token) every token reads the whole context again and every score is a
// shuffle reduction: 131 us a layer for eight tokens of a 64-head model behind 2048. Here the tokens x query heads of one key /
// value head are the rows of a tile, as in a matrix product: 16, 32, 48 or 64 rows x 32 keys per step, keys and values in turn through a ring of three
// tiles (cp.async), scores and weighted sums from 4 x 4 and 4 x 16 register blocks of packed f32 (fma.rn.f32x2: half the instructions, the
// same rate). A layer, in a graph, before (4 x 2 and 4 x 8 blocks, always 64 rows, join of a warp a vector) and now: eight tokens behind 2048, 64
// heads 33.7 and 27.8 us, 32 heads 31.9 and 21.4; 40 heads behind 4096 53.7 and 39.1; 256 tokens of 32 heads at the start 54.3 and 45.5, behind 1000
// 334 and 175. Error against 64 bits 4.6e-7 and 3.1e-7 (shorter chains). What bounds it: the f32 pipe, 38 % of it over a long prompt, with two
// warps a scheduler for the latencies of shared memory; 8 x 8 blocks, a quarter of the dimensions a warp, gained 5 % there and lost 20 % at 2048.
#include <algorithm>
#include <type_traits>

#include "attn_body.cuh"
#include "common.cuh"
#include "glue.cuh"
#include "packed_f32.cuh"

namespace alice {
namespace {

constexpr uint32_t AT_THREADS = 128, AT_KEYS = 32, AT_PITCH = 132, AT_PPITCH = 2 * AT_KEYS + 4;   // pitches in floats: rows 16 bytes apart modulo 128, so 8 rows fill the banks
constexpr uint32_t AT_TILE = AT_KEYS * AT_PITCH, AT_RING = 3;
constexpr uint32_t at_smem(uint32_t rows) { return (rows * AT_PITCH + AT_RING * AT_TILE + rows * AT_PPITCH) * 4; }

// Four f32 as two pairs.
struct F2x2 { uint64_t a, b; };
__device__ __forceinline__ F2x2 lds_2x2(uint32_t at) {
    F2x2 v;
    asm volatile("ld.shared.v2.b64 {%0,%1}, [%2];" : "=l"(v.a), "=l"(v.b) : "r"(at));
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

// One share (maximum, sum; sums of four dimensions) of a row into sums relative to the maximum M. A share without a maximum: nothing seen (all
// zeros), or nothing but NaN, which stays.
__device__ __forceinline__ void add_share(float& L, float4& A, float2 ml, float4 v, float M) {
    const float c = ml.x == -INFINITY ? 0.0f : expf(ml.x - M);
    L += ml.y * c;
    A.x += v.x * c; A.y += v.y * c; A.z += v.z * c; A.w += v.w * c;
}
// The sums from maximum M to mx >= M.
__device__ __forceinline__ void add_share(float& M, float& L, float4& A, float mx) {
    const float c = M == mx ? 1.0f : expf(M - mx);
    L *= c;
    A.x *= c; A.y *= c; A.z *= c; A.w *= c;
    M = mx;
}

// blockIdx: key / value head, tile of 16 I (token, head) rows, share of the tile's positions. cs > 1: the nsplit = cs shares are a cluster, which adds
// them up in rank order; cs = 1: each of more than one share leaves (max, sum, sums) in a.part[row][share].
template <int I>
__global__ void __launch_bounds__(AT_THREADS, 2) attn_tile_kernel(const __grid_constant__ AttnArgs a, uint32_t batch, uint32_t cs) {
    extern __shared__ __align__(16) float sm[];
    constexpr uint32_t ROWS = 16 * I;
    float* sq = sm;
    float* ring = sq + ROWS * AT_PITCH;              // keys and values of a step in turn
    float* sp = ring + AT_RING * AT_TILE;            // [rows][keys] weights, each twice
    const AttnShape s = a.shape;
    const uint32_t group = s.num_heads / s.num_kv_heads, nrows = batch * group;
    const uint32_t kvh = blockIdx.x, row0 = (gridDim.y - 1 - blockIdx.y) * ROWS, split = blockIdx.z;      // the longest first
    const uint32_t tid = threadIdx.x, tx = tid & 7, ty = tid >> 3, kv_dim = s.num_kv_heads * 128;
    const uint32_t qkv_stride = (s.num_heads + 2 * s.num_kv_heads) * 128;
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t pos0 = (uint32_t)*a.pos;
    const uint32_t seen = pos0 + min(batch, (row0 + ROWS - 1) / group + 1);      // positions the last row of the tile sees
    const uint32_t total = (seen + AT_KEYS - 1) / AT_KEYS;                        // steps, shared evenly
    const uint32_t t0 = total * split / a.nsplit * AT_KEYS, t1 = min(seen, total * (split + 1) / a.nsplit * AT_KEYS);
    const uint32_t steps = t1 > t0 ? (t1 - t0 + AT_KEYS - 1) / AT_KEYS : 0u;

    auto fetch = [&](uint32_t n) {                   // keys (n even) or values of step n / 2
        if (n < 2 * steps) {
            const uint32_t tb = t0 + (n >> 1) * AT_KEYS, to = smem_u32(ring + n % AT_RING * AT_TILE);
            const float* from = (n & 1 ? a.vcache : a.kcache) + kvh * 128 + (tid & 31) * 4;
#pragma unroll
            for (uint32_t r = tid >> 5; r < AT_KEYS; r += AT_THREADS / 32)
                cp16(to + (r * AT_PITCH + (tid & 31) * 4) * 4, from + (size_t)min(tb + r, t1 - 1) * kv_dim);      // keys past the share are masked
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (uint32_t r = tid >> 5; r < ROWS; r += AT_THREADS / 32) {
        const uint32_t row = min(row0 + r, nrows - 1), c = (tid & 31) * 4;
        cp16(smem_u32(sq + r * AT_PITCH + c), a.qkv + (size_t)(row / group) * qkv_stride + (kvh * group + row % group) * 128 + c);
    }
    fetch(0);
    fetch(1);

    const float inv_sqrt_d = __fdiv_rn(1.0f, sqrtf(128.0f));
    float m[I], l[I];
    uint64_t o[I][8];                               // dimensions 4 tx + 32 d .., two at a time
    uint32_t last[I];                               // first position the row does not see
    const uint32_t all_see = min(t1, pos0 + row0 / group + 1);      // positions below it are seen by every row of the tile
#pragma unroll
    for (int i = 0; i < I; i++) {
        m[i] = -INFINITY; l[i] = 0.0f;
        last[i] = min(t1, pos0 + (row0 + ty + 16 * i) / group + 1);
#pragma unroll
        for (int d = 0; d < 8; d++) o[i][d] = 0;
    }
    const uint32_t qa = smem_u32(sq + ty * AT_PITCH), pa = smem_u32(sp + ty * AT_PPITCH);
    for (uint32_t step = 0; step < steps; step++) {
        const uint32_t tb = t0 + step * AT_KEYS;
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                             // keys are in; the values of the step before are done with
        fetch(2 * step + 2);
        const uint32_t ka = smem_u32(ring + 2 * step % AT_RING * AT_TILE + tx * AT_PITCH);
        uint64_t acc[I][4] = {};                     // even and odd dimensions
#pragma unroll 4
        for (uint32_t c = 0; c < 32; c++) {
            F2x2 k[4];
#pragma unroll
            for (int j = 0; j < 4; j++) k[j] = lds_2x2(ka + j * 8 * AT_PITCH * 4 + c * 16);
#pragma unroll
            for (int i = 0; i < I; i++) {
                const F2x2 q = lds_2x2(qa + i * 16 * AT_PITCH * 4 + c * 16);
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fma2(q.b, k[j].b, fma2(q.a, k[j].a, acc[i][j]));
            }
        }
#pragma unroll
        for (int i = 0; i < I; i++) {
            float sc[4], mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 h = unpack2(acc[i][j]);
                sc[j] = tb + tx + 8 * j < last[i] ? (h.x + h.y) * inv_sqrt_d : -INFINITY;
                mx = fmaxf(mx, sc[j]);
            }
#pragma unroll
            for (int w = 4; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
            const float mn = fmaxf(m[i], mx);
            const float corr = m[i] == mn ? 1.0f : expf(m[i] - mn);        // a row that has seen nothing: -inf == -inf
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float p = sc[j] == -INFINITY ? 0.0f : expf(sc[j] - mn);
                *reinterpret_cast<float2*>(sp + (ty + 16 * i) * AT_PPITCH + 2 * (tx + 8 * j)) = make_float2(p, p);
                sum += p;
            }
#pragma unroll
            for (int w = 4; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
            l[i] = l[i] * corr + sum;
            m[i] = mn;
            const uint64_t c2 = pack2(corr, corr);
#pragma unroll
            for (int d = 0; d < 8; d++) o[i][d] = mul2(o[i][d], c2);
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                             // values are in, the keys done with (the weights of a row are its eight lanes' own)
        fetch(2 * step + 3);
        const uint32_t va = smem_u32(ring + (2 * step + 1) % AT_RING * AT_TILE + tx * 4);
        auto weigh = [&](auto masked) {
#pragma unroll 2
            for (uint32_t t = 0; t < AT_KEYS; t += 2) {
                F2x2 p[I];
#pragma unroll
                for (int i = 0; i < I; i++) p[i] = lds_2x2(pa + i * 16 * AT_PPITCH * 4 + t * 8);
#pragma unroll
                for (int j = 0; j < 2; j++)
#pragma unroll
                    for (int d = 0; d < 4; d++) {
                        const F2x2 v = lds_2x2(va + (t + j) * AT_PITCH * 4 + d * 128);
#pragma unroll
                        for (int i = 0; i < I; i++) {
                            if (masked.value && tb + t + j >= last[i]) continue;      // a value the row does not see may be infinite: 0 times it is not 0
                            o[i][2 * d] = fma2(j ? p[i].b : p[i].a, v.a, o[i][2 * d]);
                            o[i][2 * d + 1] = fma2(j ? p[i].b : p[i].a, v.b, o[i][2 * d + 1]);
                        }
                    }
            }
        };
        if (tb + AT_KEYS <= all_see) weigh(std::false_type{}); else weigh(std::true_type{});
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    auto output = [&](uint32_t row) { return a.attn_out + (size_t)(row / group) * a.out_stride + (size_t)(kvh * group + row % group) * 128; };
    if (cs == 1) {
#pragma unroll
        for (int i = 0; i < I; i++) {
            const uint32_t row = row0 + ty + 16 * i;
            if (row >= nrows) continue;
            float* out = output(row);
            float f = l[i] > 0.0f ? 1.0f / l[i] : 0.0f;
            if (a.nsplit > 1) {
                out = a.part + (((size_t)(row / group) * s.num_heads + kvh * group + row % group) * a.nsplit + split) * 132;
                if (tx == 0) { out[0] = m[i]; out[1] = l[i]; }
                out += 4;
                f = 1.0f;
            }
#pragma unroll
            for (int d = 0; d < 4; d++) {
                const float2 x = unpack2(o[i][2 * d]), y = unpack2(o[i][2 * d + 1]);
                reinterpret_cast<float4*>(out)[8 * d + tx] = make_float4(x.x * f, x.y * f, y.x * f, y.y * f);
            }
        }
        return;
    }
    __syncthreads();                                 // the queries are done with: the sums take their place
#pragma unroll
    for (int i = 0; i < I; i++) {
        float* out = sq + (ty + 16 * i) * AT_PITCH;
        if (tx == 0) { out[128] = m[i]; out[129] = l[i]; }
#pragma unroll
        for (int d = 0; d < 4; d++) {
            const float2 x = unpack2(o[i][2 * d]), y = unpack2(o[i][2 * d + 1]);
            reinterpret_cast<float4*>(out)[8 * d + tx] = make_float4(x.x, x.y, y.x, y.y);
        }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t lane = tid & 31;
    for (uint32_t r = split + cs * (tid >> 5); r < ROWS && row0 + r < nrows; r += cs * (AT_THREADS / 32)) {      // a warp a row, four dimensions a lane
        float2 ml[8];
        float4 v[8];
        float M = -INFINITY;
#pragma unroll
        for (uint32_t q = 0; q < 8; q++) {
            uint32_t at;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(sq + r * AT_PITCH)), "r"(q < cs ? q : 0u));
            asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];" : "=f"(ml[q].x), "=f"(ml[q].y) : "r"(at + 512) : "memory");
            asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[q].x), "=f"(v[q].y), "=f"(v[q].z), "=f"(v[q].w) : "r"(at + lane * 16) : "memory");
            M = fmaxf(M, ml[q].x);
        }
        float L = 0.0f;
        float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (uint32_t q = 0; q < 8; q++)
            if (q < cs) add_share(L, A, ml[q], v[q], M);
        const float f = L > 0.0f ? 1.0f / L : 0.0f;
        reinterpret_cast<float4*>(output(row0 + r))[lane] = make_float4(A.x * f, A.y * f, A.z * f, A.w * f);
    }
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");      // no CTA leaves while others read its sums
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}

// Joins the shares of one (token, head): four warps, every fourth share a warp's, four dimensions a lane.
__global__ void __launch_bounds__(128) attn_join_kernel(const __grid_constant__ AttnArgs a) {
    __shared__ float2 ml_[4];
    __shared__ float4 sum_[4][32];
    const uint32_t i = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_launch_dependents();
    pdl_wait();
    const float* part = a.part + (size_t)i * a.nsplit * 132;
    float M = -INFINITY, L = 0.0f;
    float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t sp0 = warp; sp0 < a.nsplit; sp0 += 32) {
        float2 ml[8];
        float4 v[8];
        float mx = M;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float* p = part + min(sp0 + 4 * j, a.nsplit - 1) * 132;
            ml[j] = __ldcg(reinterpret_cast<const float2*>(p));
            v[j] = __ldcg(reinterpret_cast<const float4*>(p + 4) + lane);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) mx = fmaxf(mx, ml[j].x);
        add_share(M, L, A, mx);
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (sp0 + 4 * j < a.nsplit) add_share(L, A, ml[j], v[j], M);
    }
    if (lane == 0) ml_[warp] = make_float2(M, L);
    sum_[warp][lane] = A;
    __syncthreads();
    if (warp) return;
    M = fmaxf(fmaxf(ml_[0].x, ml_[1].x), fmaxf(ml_[2].x, ml_[3].x));
    L = 0.0f;
    A = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < 4; w++) add_share(L, A, ml_[w], sum_[w][lane], M);
    const float inv = L > 0.0f ? 1.0f / L : 0.0f;
    const uint32_t k = i / a.shape.num_heads, head = i % a.shape.num_heads;
    reinterpret_cast<float4*>(a.attn_out + (size_t)k * a.out_stride + (size_t)head * 128)[lane] = make_float4(A.x * inv, A.y * inv, A.z * inv, A.w * inv);
}

template <int I>
cudaError_t launch_tile(cudaLaunchConfig_t& lc, const AttnArgs& a, uint32_t batch, uint32_t cs) {
    static bool done[64] = {};
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev >= 64 || !done[dev]) {
        err = cudaFuncSetAttribute(attn_tile_kernel<I>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)at_smem(16 * I));
        if (err != cudaSuccess) return err;
        if (dev < 64) done[dev] = true;
    }
    lc.dynamicSmemBytes = at_smem(16 * I);
    return cudaLaunchKernelEx(&lc, attn_tile_kernel<I>, a, batch, cs);
}

}  // namespace

cudaError_t launch_attention_tokens(const AttnArgs& args, float* qkv, uint32_t batch, uint32_t pos0, uint32_t part_vectors, int num_sms, cudaStream_t st, bool pdl) {
    AttnArgs a = args;
    const AttnShape& s = a.shape;
    if (s.head_dim != 128 || s.num_heads % s.num_kv_heads || a.npeers) return cudaErrorInvalidValue;
    const uint32_t group = s.num_heads / s.num_kv_heads, rows = batch * group, total = (pos0 + batch + AT_KEYS - 1) / AT_KEYS;
    // Tiles of 64 rows, smaller ones where a few steps would leave SMs without any (four layers of 8 x 4 heads, prompts of 17 and 64 tokens: 475 -> 429 us and
    // 583 -> 550; behind 500, 16 steps, of 8 x 8 heads 364 -> 372).
    auto tiles_of = [&](uint32_t per16) { return (rows + 16 * per16 - 1) / (16 * per16); };
    uint32_t per16 = std::min(4u, (rows + 15) / 16);
    while (per16 > 1 && total <= 8 && s.num_kv_heads * tiles_of(per16) * total < (uint32_t)num_sms) per16 = (per16 + 1) / 2;
    const uint32_t tiles = tiles_of(per16);
    if (group != 1 && group != 2 && group != 4 && group != 5 && group != 8) return cudaErrorInvalidValue;
    // Shares of the positions: two CTAs an SM. Up to eight are a cluster, which adds up by itself (11.8 against 14.5 us for 2 tokens behind 500), of a power
    // of two: rather an empty share than two steps in one (four layers of 8 x 4 heads, eight tokens behind 200, seven steps: 278 us with eight, 312 with four); more go
    // through the scratch and a join, since clusters leave slots empty when the chip is full (64 heads behind 2048, 33 shares: clusters of
    // 2 and 4 34 and 48 us, none 27.8), as many of them as the scratch holds (two key / value heads of 8, eight tokens behind 8000: 315 us for four
    // layers, 882 in clusters). Where it holds no more than a cluster has (prompts), clusters again: 45 us for 256 tokens, 63 with one share.
    const uint32_t slots = std::max(1u, 2 * (uint32_t)num_sms / (s.num_kv_heads * tiles)), room = part_vectors / (batch * s.num_heads);
    const uint32_t most = room > 8 ? std::min(slots, room) : slots, steps = (total + most - 1) / most, n = (total + steps - 1) / steps;
    uint32_t cs = 1;
    if (n <= 8 || room <= 8) while (cs < 8 && cs < total && 2 * cs <= slots) cs *= 2;
    a.nsplit = cs > 1 ? cs : n;
    cudaLaunchConfig_t lc = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = cs;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at + 1; lc.numAttrs = pdl ? 1 : 0; lc.stream = st; lc.blockDim = dim3(256);
    lc.gridDim = dim3(((s.num_heads + 2 * s.num_kv_heads) * batch + 7) / 8);
    cudaError_t err = cudaLaunchKernelEx(&lc, attn_append_kernel, a, qkv, batch);
    if (err != cudaSuccess) return err;
    lc.gridDim = dim3(s.num_kv_heads, tiles, a.nsplit); lc.blockDim = dim3(AT_THREADS);
    if (cs > 1) { lc.attrs = at; lc.numAttrs++; }
    switch (per16) {
        case 1: err = launch_tile<1>(lc, a, batch, cs); break;
        case 2: err = launch_tile<2>(lc, a, batch, cs); break;
        case 3: err = launch_tile<3>(lc, a, batch, cs); break;
        default: err = launch_tile<4>(lc, a, batch, cs);
    }
    if (err != cudaSuccess || cs > 1 || a.nsplit == 1) return err;
    lc.attrs = at + 1; lc.numAttrs = pdl ? 1 : 0;
    lc.gridDim = dim3(batch * s.num_heads); lc.blockDim = dim3(128); lc.dynamicSmemBytes = 0;
    return cudaLaunchKernelEx(&lc, attn_join_kernel, a);
}

}  // namespace alice

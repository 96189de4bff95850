// Device body of the fused decode attention: RoPE + KV append + split-KV GQA attention + split combine, for one token. Arithmetic: ALICE-LLM src/llama3.rs apply_rope :5323-5333,
// :5367-5378, KvCache::append :4773, gqa_attention :5431-5690, evaluated as an online softmax over KV splits.
#pragma once
#include "common.cuh"
#include "glue.cuh"
#include "publish.cuh"
#include "q8k.cuh"

namespace alice {

struct RopeCoef { float sn[4], cs[4]; };
// Rotation table of one position: tab[2*j] = sin, tab[2*j + 1] = cos of pos * freq[j], j = 0 .. head_dim/2 - 1
// (head_dim = 128). freq[j] = 1 / theta^(2j / head_dim) is computed on the HOST at model creation with the same libm
// powf the CPU path uses: at a position of several thousand a one-ulp difference in freq already moves the angle by
// ~1e-3 rad, which the attention scores amplify. The table depends on the position only, so it is computed once per
// decode step (by the embedding stage) and every layer's attention reads it.
__device__ __forceinline__ void rope_table_entry(float* tab, uint32_t j, uint32_t pos, const float* __restrict__ freq) {
    float sn, cs;
    sincosf(__fmul_rn((float)pos, __ldg(freq + j)), &sn, &cs);
    tab[2 * j] = sn; tab[2 * j + 1] = cs;
}
// sin / cos of the rotation angles of the 4 dims a lane owns, fetched from the table (L2 reads: another
// SM wrote it). Pairs layout: dims 4*lane + i belong to pair 2*lane + i/2; NeoX: pair 4*(lane & 15) + i.
__device__ __forceinline__ RopeCoef rope_coef(const float* __restrict__ tab, uint32_t lane, int neox) {
    RopeCoef c;
    if (!neox) {
        const float4 t = __ldcg(reinterpret_cast<const float4*>(tab) + lane);   // pairs 2*lane, 2*lane + 1
        c.sn[0] = c.sn[1] = t.x; c.cs[0] = c.cs[1] = t.y;
        c.sn[2] = c.sn[3] = t.z; c.cs[2] = c.cs[3] = t.w;
    } else {
        const float4 t0 = __ldcg(reinterpret_cast<const float4*>(tab) + 2 * (lane & 15));
        const float4 t1 = __ldcg(reinterpret_cast<const float4*>(tab) + 2 * (lane & 15) + 1);
        c.sn[0] = t0.x; c.cs[0] = t0.y; c.sn[1] = t0.z; c.cs[1] = t0.w;
        c.sn[2] = t1.x; c.cs[2] = t1.y; c.sn[3] = t1.z; c.cs[3] = t1.w;
    }
    return c;
}
__device__ __forceinline__ float4 rope4(float4 v, uint32_t lane, const RopeCoef& c, int neox) {
    float r[4] = {v.x, v.y, v.z, v.w}, out[4];
    if (!neox) {
#pragma unroll
        for (int p = 0; p < 2; p++) {
            const float x0 = r[2 * p], x1 = r[2 * p + 1];
            out[2 * p] = __fsub_rn(__fmul_rn(x0, c.cs[2 * p]), __fmul_rn(x1, c.sn[2 * p]));
            out[2 * p + 1] = __fadd_rn(__fmul_rn(x0, c.sn[2 * p]), __fmul_rn(x1, c.cs[2 * p]));
        }
    } else {
        const bool upper = lane >= 16;   // dims 64..127 are the second element of their pair
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float other = __shfl_xor_sync(0xffffffffu, r[i], 16);
            const float x0 = upper ? other : r[i], x1 = upper ? r[i] : other;
            out[i] = upper ? __fadd_rn(__fmul_rn(x0, c.sn[i]), __fmul_rn(x1, c.cs[i]))
                           : __fsub_rn(__fmul_rn(x0, c.cs[i]), __fmul_rn(x1, c.sn[i]));
        }
    }
    return make_float4(out[0], out[1], out[2], out[3]);
}

// GQA decode attention of one token with RoPE, KV append and the join of the shares fused in. One CTA an SM = one key / value head x one
// share of the positions, whose GROUP = num_heads / num_kv_heads query heads share every row it reads.
//
// What bounds it is latency: 17 MB of rows take 3 us, the chain wait -> rows -> scores -> softmax -> sums -> join the rest. So the rows go by
// cp.async into a ring of three chunks of 64 positions (a share behind 2048 positions is in flight at once), a position's score is a sum over
// 8 or 16 lanes instead of a warp's, a chunk's softmax is taken at once (one maximum and one rescaling per chunk instead of per position), and all
// warps of the last CTA take part in the join. Eight key / value heads, launches one behind the other: 4 query heads each behind 2048 positions
// 11.0 us (13.2 with a position per warp and its running maximum), 5 behind 4096 16.4 (19.9), 8 behind 2048 15.0 (22.1), 1 behind 8191
// 17.7 (20.8). Two CTAs of eight warps an SM take 11.8 / 17.5 / 15.7. Shares have at least 32 positions; CTAs without one leave at once.
constexpr int AD_WARPS = 16, AD_CHUNK = 4 * AD_WARPS, AD_STAGES = 3, AD_ROWS = AD_CHUNK / 32;
template <int GROUP>
struct AttnSmem {
    float k[AD_STAGES][AD_CHUNK][128], v[AD_STAGES][AD_CHUNK][128];
    float q[GROUP][128], newk[128], newv[128];
    float s[GROUP][AD_CHUNK], corr[GROUP], m[GROUP], l[GROUP];
    unsigned int last;
    __device__ float4* red() { return reinterpret_cast<float4*>(k); }      // sums of the warps, once the rows are used up
};

__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

template <int GROUP>
__device__ __forceinline__ void attn_decode_body(const AttnArgs& a, uint32_t kvh, uint32_t split, AttnSmem<GROUP>* sh) {
    constexpr int LP = GROUP <= 4 ? 8 : 16, NQ = 32 / LP, PW = 32 / LP;     // lanes of a position, its 16-byte pieces a lane, positions a warp takes at once
    const AttnShape s = a.shape;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t q_dim = s.num_heads * s.head_dim, kv_dim = s.num_kv_heads * s.head_dim;
    // the queries and the token's own row, asked for together with the position
    constexpr int NX = (GROUP + 2 + AD_WARPS - 1) / AD_WARPS;
    float4 own[NX];
#pragma unroll
    for (int i = 0; i < NX; i++) {
        const uint32_t h = warp + i * AD_WARPS;
        if (h < GROUP + 2) own[i] = __ldcg(reinterpret_cast<const float4*>(a.qkv + (h < GROUP ? (kvh * GROUP + h) * 128 : q_dim + (h == GROUP ? 0u : kv_dim) + kvh * 128)) + lane);
    }
    const RopeCoef rc = rope_coef(a.rope_tab, lane, a.neox);
    const uint32_t pos = (uint32_t)*a.pos;
    const uint32_t seq = pos + 1, per = max((seq + a.nsplit - 1) / a.nsplit, 32u), active = (seq + per - 1) / per;
    if (split >= active) return;
    const uint32_t t0 = split * per, t1 = min(seq, t0 + per), chunks = (t1 - t0 + AD_CHUNK - 1) / AD_CHUNK;
    const float* const kc = a.kcache + (size_t)kvh * 128;
    const float* const vc = a.vcache + (size_t)kvh * 128;

    auto fetch = [&](uint32_t c) {
        if (c < chunks) {
            const uint32_t st = c % AD_STAGES;
#pragma unroll
            for (int i = 0; i < AD_CHUNK * 32 / (AD_WARPS * 32); i++) {
                const uint32_t r = warp + i * AD_WARPS, t = t0 + c * AD_CHUNK + r;
                if (t < t1 && t < pos) {
                    cp16(smem_u32(&sh->k[st][r][lane * 4]), kc + (size_t)t * kv_dim + lane * 4);
                    cp16(smem_u32(&sh->v[st][r][lane * 4]), vc + (size_t)t * kv_dim + lane * 4);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (uint32_t c = 0; c < AD_STAGES; c++) fetch(c);
    // rotated; the own row also goes to the cache (KvCache::append, src/llama3.rs:4773)
#pragma unroll
    for (int i = 0; i < NX; i++) {
        const uint32_t h = warp + i * AD_WARPS;
        if (h >= GROUP + 2) continue;
        const float4 x = h <= GROUP ? rope4(own[i], lane, rc, a.neox) : own[i];
        reinterpret_cast<float4*>(h < GROUP ? sh->q[h] : h == GROUP ? sh->newk : sh->newv)[lane] = x;
        if (h >= GROUP && pos < t1) reinterpret_cast<float4*>((h == GROUP ? a.kcache : a.vcache) + (size_t)pos * kv_dim + kvh * 128)[lane] = x;
    }
    __syncthreads();
    const uint32_t lp = lane % LP, pw = lane / LP;
    float4 q[GROUP][NQ];
#pragma unroll
    for (int g = 0; g < GROUP; g++)
#pragma unroll
        for (int i = 0; i < NQ; i++) q[g][i] = reinterpret_cast<const float4*>(sh->q[g])[lp + LP * i];
    const float inv_sqrt_d = __fdiv_rn(1.0f, sqrtf((float)s.head_dim));
    float m = -INFINITY, l = 0.0f;              // of head `warp`
    float4 acc[GROUP];
#pragma unroll
    for (int g = 0; g < GROUP; g++) acc[g] = make_float4(0.f, 0.f, 0.f, 0.f);

    for (uint32_t c = 0; c < chunks; c++) {
        const uint32_t st = c % AD_STAGES, tb = t0 + c * AD_CHUNK, n = min((uint32_t)AD_CHUNK, t1 - tb);
        if (c) asm volatile("cp.async.wait_group %0;" ::"n"(AD_STAGES - 2) : "memory");
        else asm volatile("cp.async.wait_group %0;" ::"n"(AD_STAGES - 1) : "memory");
        __syncthreads();
        if (c) fetch(c + AD_STAGES - 1);         // into the stage of the chunk before, which every warp has left
#pragma unroll
        for (int r0 = 0; r0 < AD_CHUNK; r0 += AD_WARPS * PW) {
            const uint32_t r = r0 + warp * PW + pw;
            if (r0 + warp * PW >= n) break;
            const float4* kr = reinterpret_cast<const float4*>(tb + r == pos ? sh->newk : sh->k[st][r]);
            float sc[GROUP] = {};
#pragma unroll
            for (int i = 0; i < NQ; i++) {
                const float4 k = kr[lp + LP * i];
#pragma unroll
                for (int g = 0; g < GROUP; g++) sc[g] = fmaf(q[g][i].x, k.x, fmaf(q[g][i].y, k.y, fmaf(q[g][i].z, k.z, fmaf(q[g][i].w, k.w, sc[g]))));
            }
#pragma unroll
            for (int o = LP / 2; o > 0; o >>= 1)
#pragma unroll
                for (int g = 0; g < GROUP; g++) sc[g] += __shfl_xor_sync(0xffffffffu, sc[g], o);
            if (lp == 0)
#pragma unroll
                for (int g = 0; g < GROUP; g++) sh->s[g][r] = sc[g] * inv_sqrt_d;
        }
        __syncthreads();
        if (warp < GROUP) {
            float x[AD_ROWS], mx = m;
#pragma unroll
            for (int i = 0; i < AD_ROWS; i++) {
                const uint32_t r = lane + 32 * i;
                x[i] = r < n ? sh->s[warp][r] : -INFINITY;
                mx = fmaxf(mx, x[i]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float corr = m == mx ? 1.0f : expf(m - mx);
            float sum = 0.0f;
#pragma unroll
            for (int i = 0; i < AD_ROWS; i++) {
                x[i] = x[i] == -INFINITY ? 0.0f : expf(x[i] - mx);
                sh->s[warp][lane + 32 * i] = x[i];
                sum += x[i];
            }
            l = l * corr + warp_sum(sum);
            m = mx;
            if (lane == 0) sh->corr[warp] = corr;
        }
        __syncthreads();
        if (c) {
#pragma unroll
            for (int g = 0; g < GROUP; g++) {
                const float f = sh->corr[g];
                acc[g].x *= f; acc[g].y *= f; acc[g].z *= f; acc[g].w *= f;
            }
        }
        float p[GROUP][4];
#pragma unroll
        for (int g = 0; g < GROUP; g++) {
            const float4 x = reinterpret_cast<const float4*>(sh->s[g])[warp];
            p[g][0] = x.x; p[g][1] = x.y; p[g][2] = x.z; p[g][3] = x.w;
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t r = warp * 4 + j;
            if (r < n) {
                const float4 v = reinterpret_cast<const float4*>(tb + r == pos ? sh->newv : sh->v[st][r])[lane];
#pragma unroll
                for (int g = 0; g < GROUP; g++) {
                    acc[g].x = fmaf(p[g][j], v.x, acc[g].x); acc[g].y = fmaf(p[g][j], v.y, acc[g].y);
                    acc[g].z = fmaf(p[g][j], v.z, acc[g].z); acc[g].w = fmaf(p[g][j], v.w, acc[g].w);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float4* const red = sh->red();
#pragma unroll
    for (int g = 0; g < GROUP; g++) red[(warp * GROUP + g) * 32 + lane] = acc[g];
    if (warp < GROUP && lane == 0) { sh->m[warp] = m; sh->l[warp] = l; }
    __syncthreads();
    const uint32_t stride = s.head_dim + 4;   // (m, l, pad, pad, sums[128]): keeps the sums 16-byte aligned
    float* const part = a.part;
    float4 o_keep = make_float4(0.f, 0.f, 0.f, 0.f);      // output of head `warp`, this lane's 4 dims
    auto finish = [&](float4 A, float L) {
        const uint32_t head = kvh * GROUP + warp;
        const float inv = L > 0.0f ? 1.0f / L : 0.0f;
        o_keep = make_float4(A.x * inv, A.y * inv, A.z * inv, A.w * inv);
        reinterpret_cast<float4*>(a.attn_out + (size_t)head * 128)[lane] = o_keep;
        for (uint32_t p = 0; p < a.npeers; p++) reinterpret_cast<float4*>(a.peer_out[p] + (size_t)head * 128)[lane] = o_keep;
    };
    if (warp < GROUP) {
        float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < AD_WARPS; w++) {
            const float4 x = red[(w * GROUP + warp) * 32 + lane];
            A.x += x.x; A.y += x.y; A.z += x.z; A.w += x.w;
        }
        if (active == 1) {
            finish(A, l);
        } else {
            float* out = part + ((size_t)split * s.num_heads + kvh * GROUP + warp) * stride;
            if (lane == 0) *reinterpret_cast<float2*>(out) = make_float2(m, l);
            reinterpret_cast<float4*>(out + 4)[lane] = A;
        }
    }
    if (active > 1) {
        // the last CTA of this key / value head joins the shares
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            const unsigned int ticket = atomicAdd(a.tickets + kvh, 1u);
            sh->last = ticket == active - 1 ? 1u : 0u;
            if (sh->last) { a.tickets[kvh] = 0; __threadfence(); }      // ready for the next launch
        }
        __syncthreads();
        if (!sh->last) return;
        constexpr int WH = AD_WARPS / GROUP;             // warps of a head
        const uint32_t g = warp % GROUP, sub = warp / GROUP;
        if (sub < WH) {
            const float* base = part + (size_t)(kvh * GROUP + g) * stride;
            const size_t step = (size_t)s.num_heads * stride;
            float ms[2], ls[2], M = -INFINITY;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint32_t sp = lane + 32 * i;
                const float2 ml = sp < active ? __ldcg(reinterpret_cast<const float2*>(base + sp * step)) : make_float2(-INFINITY, 0.0f);
                ms[i] = ml.x; ls[i] = ml.y;
                M = fmaxf(M, ms[i]);
            }
            constexpr int SB = 8;                        // sums fetched at once
            float4 x[SB];
            auto load = [&](uint32_t sp0) {
#pragma unroll
                for (int j = 0; j < SB; j++) x[j] = __ldcg(reinterpret_cast<const float4*>(base + min(sp0 + j * WH, active - 1) * step + 4) + lane);
            };
            load(sub);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
            float cs[2], L = 0.0f;
#pragma unroll
            for (int i = 0; i < 2; i++) { cs[i] = ms[i] == -INFINITY ? 0.0f : expf(ms[i] - M); L += ls[i] * cs[i]; }
            L = warp_sum(L);
            float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
            for (uint32_t sp0 = sub; sp0 < active; sp0 += SB * WH) {
                if (sp0 != sub) load(sp0);
#pragma unroll
                for (int j = 0; j < SB; j++) {
                    const uint32_t sp = sp0 + j * WH;
                    const float f = __shfl_sync(0xffffffffu, sp < 32 ? cs[0] : cs[1], sp & 31);
                    if (sp < active) { A.x += x[j].x * f; A.y += x[j].y * f; A.z += x[j].z * f; A.w += x[j].w * f; }
                }
            }
            red[(sub * GROUP + g) * 32 + lane] = A;
            if (sub == 0 && lane == 0) sh->l[g] = L;
        }
        __syncthreads();
        if (warp < GROUP) {
            float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < WH; w++) {
                const float4 y = red[(w * GROUP + warp) * 32 + lane];
                A.x += y.x; A.y += y.y; A.z += y.z; A.w += y.w;
            }
            finish(A, sh->l[warp]);
        }
    }
    if (a.q8.qs != nullptr && (GROUP % 2) == 0) {
        // Q8_K of this KV head's GROUP * 128 outputs = GROUP / 2 whole blocks (quantize_row_q8_k, src/gguf.rs:1323): the
        // outputs go through shared memory so that a warp sees the two heads of its block
        if (warp < GROUP) reinterpret_cast<float4*>(sh->q[warp])[lane] = o_keep;
        __syncthreads();
        if (warp < GROUP / 2) {
            const size_t blk = (kvh * GROUP) / 2 + warp;
            const int hsel = 2 * (int)warp + (int)(lane >> 4);
            Q8KLaneInput in;
            in.a = reinterpret_cast<const float4*>(sh->q[hsel])[(lane & 15) * 2];
            in.b = reinterpret_cast<const float4*>(sh->q[hsel])[(lane & 15) * 2 + 1];
            q8k_quantize_block_warp(in, lane, a.q8.qs + blk * QK_K, a.q8.d + blk, a.q8.bsums + blk * 16);
        }
    }
}

}  // namespace alice

// 16-row tiles of K-quant weights times up to eight Q8_K vectors on the int8 tensor cores (csrc/gemv_kq_rows.cu, and the digits of
// the activation sums for csrc/gemm_kq.cu).
//
// The speculative-verify step feeds 4..8 tokens through every projection. The weights are streamed and unpacked ONCE:
// a warp owns a tile of 16 rows (mma M), the unpacked 4/5/6-bit quants of a 32-element sub-block are the A operand
// (u8, 16 rows x 32) of one mma.sync m16n8k32 and the Q8_K int8 activations of the up-to-8 input vectors are the B
// operand (32 x 8 columns = the batch), so one instruction yields the integer sub-block dot products of 16 rows x 8
// vectors. Per-sub-block scales are applied to the int32 results as in q4k_q8k_dot (src/gguf.rs:3201-3251); the
// min term sum_is m[is] * bsum[is] is one more pair of small MMAs (A = the 6-bit mins, B = the sub-block sums of the
// activations split into two signed base-64 digits). The reference does the same on the GPU with
// dequant_matvec_q4k_batch4.wgsl / swiglu_fused_q4k_batch4.wgsl (weights decoded once for 4 inputs, in f32).
#pragma once
#include "gemv_mma.cuh"

namespace alice {

struct KqActs {
    uint32_t qs;      // shared address of int8 [8][xs]
    uint32_t xs;      // bytes between vectors
    uint32_t d;       // shared address of f32 [8][nb]
    uint32_t bsd;     // shared address of s8 [8][nb][16]: base-64 digits of the 8 sub-block (32-element) sums, low digits in bytes 0..7, high in 8..15
    uint32_t bs16;    // shared address of s8 [8][nb][32]: base-64 digits of the 16 sub-block (16-element) sums, low 0..15, high 16..31 (Q6_K)
    uint32_t nb;
};
__device__ __forceinline__ void mma_s8s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0));
}

__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
// Signed base-64 digits (v = 64 hi + lo) of a token's activation sums: K4 the 8 sums of 32 (lo 0..7 | hi 8..15), Q6_K the 16 sums of 16.
template <bool Q6>
__device__ __forceinline__ void kq_store_digits(uint32_t at, const uint4& s0, const uint4& s1) {
    const uint32_t w[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    constexpr int NV = Q6 ? 16 : 8;
    uint32_t lo[NV / 4] = {}, hi[NV / 4] = {};
#pragma unroll
    for (int i = 0; i < NV; i++) {
        int v;
        if (Q6) v = (int)(int16_t)(i & 1 ? w[i >> 1] >> 16 : w[i >> 1] & 0xffffu);
        else v = (int)(int16_t)(w[i] & 0xffffu) + (int)(int16_t)(w[i] >> 16);
        const int l = ((v + 32) & 63) - 32, h = (v - l) >> 6;
        lo[i >> 2] |= (uint32_t)(l & 0xff) << (8 * (i & 3));
        hi[i >> 2] |= (uint32_t)(h & 0xff) << (8 * (i & 3));
    }
#pragma unroll
    for (int i = 0; i < NV / 4; i++) { sts32(at + 4 * i, lo[i]); sts32(at + NV + 4 * i, hi[i]); }
}

// 6-bit scales (sc) and mins (m) of a K4 header as four words of four bytes each: sub-blocks 0..3 and 4..7
// (get_scale_min_k4, src/gguf.rs:794-802).
__device__ __forceinline__ void k4_unpack(const uint4& h, uint32_t& sc_lo, uint32_t& sc_hi, uint32_t& m_lo, uint32_t& m_hi) {
    sc_lo = h.y & 0x3f3f3f3fu;
    m_lo = h.z & 0x3f3f3f3fu;
    sc_hi = (h.w & 0x0f0f0f0fu) | ((h.y >> 2) & 0x30303030u);
    m_hi = ((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u);
}

// Thread (g = lane / 4, t = lane % 4) of a tile holds outputs (row g, vectors 2t, 2t+1) and (row g + 8, vectors 2t, 2t+1).
// k slot mapping of one 32-element sub-block: slots 4t..4t+3 = elements 8t..8t+3, slots 16+4t..16+4t+3 = elements
// 8t+4..8t+7, so a thread's A bytes are 8 consecutive weight bytes and its B bytes 8 consecutive activations.

// ── Q4_K / Q5_K tile: blocks [b_lo, b_hi) of rows rowA (g) and rowB (g + 8).
template <bool Q5>
struct KqK4 {
    static constexpr uint32_t BLOCK_BYTES = Q5 ? 176 : 144;
    __device__ static void tile(uint32_t rowA, uint32_t rowB, uint32_t b_lo, uint32_t b_hi, const KqActs& x, uint32_t lane, float (&acc)[4]) {
        const uint32_t t = lane & 3u, g = lane >> 2;
        constexpr uint32_t LO = 0x0f0f0f0fu;
        constexpr uint32_t QS = Q5 ? 48u : 16u;
        for (uint32_t blk = b_lo; blk < b_hi; blk++) {
            const uint32_t pA = rowA + blk * BLOCK_BYTES, pB = rowB + blk * BLOCK_BYTES;
            const uint4 hA = lds128(pA), hB = lds128(pB);
            uint32_t scA_lo, scA_hi, mA_lo, mA_hi, scB_lo, scB_hi, mB_lo, mB_hi;
            k4_unpack(hA, scA_lo, scA_hi, mA_lo, mA_hi);
            k4_unpack(hB, scB_lo, scB_hi, mB_lo, mB_hi);
            uint2 qhA = make_uint2(0u, 0u), qhB = make_uint2(0u, 0u);
            if (Q5) { qhA = lds64(pA + 16 + 8 * t); qhB = lds64(pB + 16 + 8 * t); }
            const uint32_t xq = x.qs + g * x.xs + blk * 256 + 8 * t;
            int tot[4] = {0, 0, 0, 0};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint2 wA = lds64(pA + QS + 32 * j + 8 * t), wB = lds64(pB + QS + 32 * j + 8 * t);
                const uint2 xl = lds64(xq + 64 * j), xh = lds64(xq + 64 * j + 32);
                uint32_t a0 = wA.x & LO, a1 = wB.x & LO, a2 = wA.y & LO, a3 = wB.y & LO;
                uint32_t e0 = (wA.x >> 4) & LO, e1 = (wB.x >> 4) & LO, e2 = (wA.y >> 4) & LO, e3 = (wB.y >> 4) & LO;
                if (Q5) {
                    constexpr uint32_t B0 = 0x01010101u;
                    a0 |= ((qhA.x >> (2 * j)) & B0) << 4; a1 |= ((qhB.x >> (2 * j)) & B0) << 4;
                    a2 |= ((qhA.y >> (2 * j)) & B0) << 4; a3 |= ((qhB.y >> (2 * j)) & B0) << 4;
                    e0 |= ((qhA.x >> (2 * j + 1)) & B0) << 4; e1 |= ((qhB.x >> (2 * j + 1)) & B0) << 4;
                    e2 |= ((qhA.y >> (2 * j + 1)) & B0) << 4; e3 |= ((qhB.y >> (2 * j + 1)) & B0) << 4;
                }
                int cl[4] = {0, 0, 0, 0}, ch[4] = {0, 0, 0, 0};
                mma_u8s8_k32(cl, a0, a1, a2, a3, xl.x, xl.y);
                mma_u8s8_k32(ch, e0, e1, e2, e3, xh.x, xh.y);
                // sub-blocks 2j (low nibbles) and 2j + 1 (high nibbles)
                const uint32_t wAs = j < 2 ? scA_lo : scA_hi, wBs = j < 2 ? scB_lo : scB_hi;
                const int sA0 = (int)((wAs >> (16 * (j & 1))) & 0xffu), sA1 = (int)((wAs >> (16 * (j & 1) + 8)) & 0xffu);
                const int sB0 = (int)((wBs >> (16 * (j & 1))) & 0xffu), sB1 = (int)((wBs >> (16 * (j & 1) + 8)) & 0xffu);
                tot[0] += sA0 * cl[0] + sA1 * ch[0]; tot[1] += sA0 * cl[1] + sA1 * ch[1];
                tot[2] += sB0 * cl[2] + sB1 * ch[2]; tot[3] += sB0 * cl[3] + sB1 * ch[3];
            }
            // min term: sum over the 8 sub-blocks of m[is] * (sum of the 32 activations), k slots 0..7 = sub-blocks
            const uint32_t aM0 = t == 0 ? mA_lo : (t == 1 ? mA_hi : 0u), aM1 = t == 0 ? mB_lo : (t == 1 ? mB_hi : 0u);
            const uint32_t dg = x.bsd + (g * x.nb + blk) * 16;
            const uint32_t bl = t < 2 ? lds32(dg + 4 * t) : 0u, bh = t < 2 ? lds32(dg + 8 + 4 * t) : 0u;
            int sm[4] = {0, 0, 0, 0};
            mma_u8s8_k16(sm, aM0, aM1, bh);
#pragma unroll
            for (int i = 0; i < 4; i++) sm[i] <<= 6;
            mma_u8s8_k16(sm, aM0, aM1, bl);
            const float2 dmA = __half22float2(*reinterpret_cast<const __half2*>(&hA.x));
            const float2 dmB = __half22float2(*reinterpret_cast<const __half2*>(&hB.x));
            const float d80 = ldsf(x.d + ((2 * t) * x.nb + blk) * 4), d81 = ldsf(x.d + ((2 * t + 1) * x.nb + blk) * 4);
            acc[0] += (dmA.x * d80) * (float)tot[0] - (dmA.y * d80) * (float)sm[0];
            acc[1] += (dmA.x * d81) * (float)tot[1] - (dmA.y * d81) * (float)sm[1];
            acc[2] += (dmB.x * d80) * (float)tot[2] - (dmB.y * d80) * (float)sm[2];
            acc[3] += (dmB.x * d81) * (float)tot[3] - (dmB.y * d81) * (float)sm[3];
        }
    }
};

// ── Q6_K tile: 210-byte blocks ql[128] qh[64] sc[16] d (src/gguf.rs:1205-1246); integer dot as q6k_q8k_dot
// (src/gguf.rs:3282-3319): sum over the 16 sub-blocks of 16 elements of sc[is] * dot(q - 32, q8). The -32 goes through
// the activation sums: sc * (dot(q, q8) - 32 * bsum[is]); the bias sum_is sc[is] * bsum[is] is a pair of s8 x s8 MMAs.
// Blocks are only 2-byte aligned in a row, so words are fetched as two aligned halves and funnel-shifted.
// A thread covers, for half n and 16-column group i, the columns l = 16 i + 4 t .. + 3 of all four quadrants: one ql
// word serves quadrants 0 / 2 (low / high nibbles), one serves 1 / 3, one qh word carries the two high bits of all four.
struct KqQ6K {
    static constexpr uint32_t BLOCK_BYTES = 210;
    __device__ static void tile(uint32_t rowA, uint32_t rowB, uint32_t b_lo, uint32_t b_hi, const KqActs& x, uint32_t lane, float (&acc)[4]) {
        const uint32_t t = lane & 3u, g = lane >> 2;
        constexpr uint32_t LO = 0x0f0f0f0fu, H2 = 0x30303030u;
        for (uint32_t blk = b_lo; blk < b_hi; blk++) {
            const uint32_t pA = rowA + blk * BLOCK_BYTES, pB = rowB + blk * BLOCK_BYTES;
            const uint32_t xq = x.qs + g * x.xs + blk * 256 + 4 * t;
            int tot[4] = {0, 0, 0, 0};
#pragma unroll
            for (int n = 0; n < 2; n++) {
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const uint32_t o = 16 * i + 4 * t;
                    const uint32_t lA0 = lds32_u2(pA + 64 * n + o), lA1 = lds32_u2(pA + 64 * n + 32 + o), hA = lds32_u2(pA + 128 + 32 * n + o);
                    const uint32_t lB0 = lds32_u2(pB + 64 * n + o), lB1 = lds32_u2(pB + 64 * n + 32 + o), hB = lds32_u2(pB + 128 + 32 * n + o);
                    // the four int8 scales of this (n, i): index 8n + i + {0, 2, 4, 6}
                    const uint32_t sa = lds32_u2(pA + 192 + 8 * n) >> (8 * i), sa2 = lds32_u2(pA + 196 + 8 * n) >> (8 * i);
                    const uint32_t sb = lds32_u2(pB + 192 + 8 * n) >> (8 * i), sb2 = lds32_u2(pB + 196 + 8 * n) >> (8 * i);
                    const int scA[4] = {(int)(int8_t)(sa & 0xff), (int)(int8_t)((sa >> 16) & 0xff), (int)(int8_t)(sa2 & 0xff), (int)(int8_t)((sa2 >> 16) & 0xff)};
                    const int scB[4] = {(int)(int8_t)(sb & 0xff), (int)(int8_t)((sb >> 16) & 0xff), (int)(int8_t)(sb2 & 0xff), (int)(int8_t)((sb2 >> 16) & 0xff)};
                    const uint32_t qa[4] = {(lA0 & LO) | ((hA << 4) & H2), (lA1 & LO) | ((hA << 2) & H2), ((lA0 >> 4) & LO) | (hA & H2), ((lA1 >> 4) & LO) | ((hA >> 2) & H2)};
                    const uint32_t qb[4] = {(lB0 & LO) | ((hB << 4) & H2), (lB1 & LO) | ((hB << 2) & H2), ((lB0 >> 4) & LO) | (hB & H2), ((lB1 >> 4) & LO) | ((hB >> 2) & H2)};
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const uint32_t bx = lds32(xq + 128 * n + 32 * q + 16 * i);
                        int c[4] = {0, 0, 0, 0};
                        mma_u8s8_k16(c, qa[q], qb[q], bx);
                        tot[0] += scA[q] * c[0]; tot[1] += scA[q] * c[1]; tot[2] += scB[q] * c[2]; tot[3] += scB[q] * c[3];
                    }
                }
            }
            // bias: 32 * sum over the 16 sub-blocks of sc[is] * bsum[is]; k slots = sub-blocks, 4t .. 4t+3 per thread
            const uint32_t aS0 = lds32_u2(pA + 192 + 4 * t), aS1 = lds32_u2(pB + 192 + 4 * t);
            const uint32_t dg = x.bs16 + (g * x.nb + blk) * 32;
            const uint32_t bl = lds32(dg + 4 * t), bh = lds32(dg + 16 + 4 * t);
            int bias[4] = {0, 0, 0, 0};
            mma_s8s8_k16(bias, aS0, aS1, bh);
#pragma unroll
            for (int i = 0; i < 4; i++) bias[i] <<= 6;
            mma_s8s8_k16(bias, aS0, aS1, bl);
            const float dA = f16_bits_to_f32(lds16(pA + 208)), dB = f16_bits_to_f32(lds16(pB + 208));
            const float d80 = ldsf(x.d + ((2 * t) * x.nb + blk) * 4), d81 = ldsf(x.d + ((2 * t + 1) * x.nb + blk) * 4);
            acc[0] += (dA * d80) * (float)(tot[0] - 32 * bias[0]);
            acc[1] += (dA * d81) * (float)(tot[1] - 32 * bias[1]);
            acc[2] += (dB * d80) * (float)(tot[2] - 32 * bias[2]);
            acc[3] += (dB * d81) * (float)(tot[3] - 32 * bias[3]);
        }
    }
};

}  // namespace alice

// K-quant products with many vectors on the int8 tensor path, with the integer arithmetic of the K-quant block dots kept as it is
// (q4k_q8k_dot src/gguf.rs:3201-3251, q6k_q8k_dot :3282-3319): quants times Q8_K activations in int32 per sub-block, times the
// 6- or 8-bit scale in int32, one f32 step per block of 256. That is why the products are mma.sync u8 x s8: scale times
// quant needs more than 8 bits, and up to 13 bits for Q6_K, more than an f16 holds.
//
// A CTA (WM x WN warps) owns 32 WM rows x 8 NTW WN tokens and walks the 256-column blocks: raw weight blocks and Q8_K blocks come
// in with cp.async one to two blocks ahead, a warp unpacks 32 rows of a sub-block into A fragments and uses them for its NTW x 8
// tokens (32: sums in int32 and f32 then leave room for two CTAs of eight warps an SM). The min / bias term is a pair of products of the scales with base-64 digits of the activation sums, once per block.
// What bounds it: the instructions around the products (eight to sixteen each), for few tokens HBM. 9 to 64 tokens; more run on tcgen05
// (csrc/gemm_kq_tc.cu). Where tiles are fewer than two per SM, a cluster shares the columns of a tile and adds its
// parts through distributed shared memory in a fixed order.
#include <algorithm>

#include "../../include/alice_cuda.h"
#include "common.cuh"
#include "gemm_kq.cuh"
#include "gemv_kq_mma.cuh"

namespace alice {
namespace {

struct KqGemmArgs {
    const uint8_t* w[3];
    uint32_t rows[3], y_off[3], tile0[4], nw;
    const uint8_t* up;
    uint32_t row_bytes, nb;
    const int8_t* qs;            // [batch][nb * 256]
    const float* d;              // [batch][nb]
    const int16_t* bsums;        // [batch][nb][16]
    float* y;
    const float* resid;
    uint32_t y_stride, batch, stages;
};

template <int FMT> struct KqBlock;      // bytes of a block, 16-byte pieces fetched per row, shared-memory pitch of a row and of a token
// pitches: 64-bit reads of 4 rows x 32 bytes (K4) or 32-bit reads of 8 rows x 16 bytes (Q6_K) fill the banks once
template <> struct KqBlock<4> { static constexpr uint32_t BB = 144, CH = 9, PITCH = 160, XP = 288, DG = 16; };
template <> struct KqBlock<5> { static constexpr uint32_t BB = 176, CH = 11, PITCH = 224, XP = 288, DG = 16; };
template <> struct KqBlock<6> { static constexpr uint32_t BB = 210, CH = 14, PITCH = 240, XP = 272, DG = 32; };

template <int FMT, int WM, int WN, int NTW>
struct KqStage {      // byte offsets inside a stage
    static constexpr uint32_t ROWS = 32 * WM, N = 8 * NTW * WN, THREADS = 32 * WM * WN, X = ROWS * KqBlock<FMT>::PITCH, D = X + N * KqBlock<FMT>::XP, DIG = D + N * 4,
                              BYTES = (DIG + N * KqBlock<FMT>::DG + 127) & ~127u;
};

__device__ __forceinline__ void cp16z(uint32_t dst, const void* src, uint32_t n) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp4z(uint32_t dst, const void* src, uint32_t n) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void mma0_u8s8_k32(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma0_u8s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
// Plain loads: the products are no volatile assembly here either, so the compiler may bring operands in ahead of earlier products.
template <class V> __device__ __forceinline__ V ld(const uint8_t* p) { return *reinterpret_cast<const V*>(p); }
__device__ __forceinline__ uint32_t ld_u2(const uint8_t* p) {      // a 32-bit word at a 2-byte boundary
    const uint32_t a = smem_u32(p) & 2u;
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p - a);
    return __funnelshift_r(q[0], q[1], a * 8u);
}

template <int FMT, int WM, int WN, int NTW, bool SW>
__global__ void __launch_bounds__(32 * WM * WN, 2) kq_gemm_kernel(const __grid_constant__ KqGemmArgs a, const uint32_t KS) {
    extern __shared__ __align__(128) uint8_t smem[];
    using B = KqBlock<FMT>;
    using St = KqStage<FMT, WM, WN, NTW>;
    constexpr uint32_t N = St::N, G_ROWS = St::ROWS, G_THREADS = St::THREADS;
    static_assert(N <= G_THREADS, "a thread per token prepares the activation sums");
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3u;
    const uint32_t wm = warp % WM, wn = warp / WM;
    const uint32_t rank = KS > 1 ? blockIdx.x % KS : 0u, tile = blockIdx.x / KS, tok0 = blockIdx.y * N;
    const uint32_t ring = smem_u32(smem);
    uint32_t s = 0;
    if (!SW) while (s + 1 < a.nw && tile >= a.tile0[s + 1]) s++;
    const uint32_t seg_rows = a.rows[s], r0 = (tile - a.tile0[s]) * (SW ? G_ROWS / 2 : G_ROWS);
    const uint64_t total = (uint64_t)seg_rows * a.row_bytes;
    const uint32_t b_lo = a.nb * rank / KS, nblk = a.nb * (rank + 1) / KS - b_lo;
    pdl_launch_dependents();
    pdl_wait();

    // row of the matrix behind row i of the stage: with SwiGLU each warp row half holds 16 gate rows, then the same 16 of up
    auto stage_row = [&](uint32_t i) { return SW ? r0 + (i >> 5) * 16 + (i & 15u) : r0 + i; };
    auto fetch = [&](uint32_t k) {
        const uint32_t st = ring + (k % a.stages) * St::BYTES, blk = b_lo + k;
#pragma unroll
        for (uint32_t i = tid; i < G_ROWS * B::CH; i += G_THREADS) {
            const uint32_t r = i / B::CH, c = i - r * B::CH, row = min(stage_row(r), seg_rows - 1);
            const uint8_t* m = SW && (r & 16u) ? a.up : a.w[s];
            const uint64_t off = (((uint64_t)row * a.row_bytes + (uint64_t)blk * B::BB) & ~(uint64_t)15) + c * 16;
            cp16z(st + r * B::PITCH + c * 16, off < total ? m + off : m, off < total ? (uint32_t)min((uint64_t)16, total - off) : 0u);
        }
#pragma unroll
        for (uint32_t i = tid; i < N * 16; i += G_THREADS) {
            const uint32_t v = i >> 4, c = i & 15u, tok = tok0 + v, ok = tok < a.batch;
            cp16z(st + St::X + v * B::XP + c * 16, a.qs + ((size_t)(ok ? tok : 0) * a.nb + blk) * 256 + c * 16, ok ? 16u : 0u);
        }
        if (tid < N) {
            const uint32_t tok = tok0 + tid, ok = tok < a.batch;
            cp4z(st + St::D + tid * 4, a.d + (size_t)(ok ? tok : 0) * a.nb + blk, ok ? 4u : 0u);
        }
    };
    uint4 s0, s1;
    auto sums = [&](uint32_t k) {      // the activation sums of block k, a token per thread
        s0 = s1 = make_uint4(0u, 0u, 0u, 0u);
        if (tid < N && tok0 + tid < a.batch && k < nblk) {
            const uint4* p = reinterpret_cast<const uint4*>(a.bsums + ((size_t)(tok0 + tid) * a.nb + b_lo + k) * 16);
            s0 = __ldcg(p); s1 = __ldcg(p + 1);
        }
    };
    for (uint32_t k = 0; k + 1 < a.stages; k++) {
        if (k < nblk) fetch(k);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    sums(0);

    float acc[2][NTW][4] = {};
    for (uint32_t k = 0; k < nblk; k++) {
        const uint32_t st = ring + (k % a.stages) * St::BYTES, blk = b_lo + k;
        if (tid < N) kq_store_digits<FMT == 6>(st + St::DIG + tid * B::DG, s0, s1);
        sums(k + 1);
        if (a.stages == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
        else asm volatile("cp.async.wait_group 1;" ::: "memory");      // 3 stages: one younger group may be in flight
        __syncthreads();                                               // block k is in; everyone is done with block k - 1
        if (k + a.stages - 1 < nblk) fetch(k + a.stages - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");

        int tot[2][NTW][4] = {};
        const uint8_t* const sp = smem + (k % a.stages) * St::BYTES;
        const uint8_t* p[2][2];      // rows g and g + 8 of both 16-row tiles
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t r = wm * 32 + m * 16 + h * 8 + g;
                p[m][h] = sp + r * B::PITCH;
                if (FMT == 6) p[m][h] += ((uint32_t)min(stage_row(r), seg_rows - 1) * a.row_bytes + blk * B::BB) & 15u;
            }
        const uint8_t* const xa = sp + St::X + (wn * NTW * 8 + g) * B::XP;
        const uint8_t* const dg = sp + St::DIG + (wn * NTW * 8 + g) * B::DG;
        if constexpr (FMT != 6) {
            constexpr uint32_t LO = 0x0f0f0f0fu, QS = FMT == 5 ? 48u : 16u;
            uint32_t sc[2][2][2];                            // [tile][row half]: scales of the sub-blocks to come, two a step
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    uint32_t mn_lo, mn_hi;
                    k4_unpack(ld<uint4>(p[m][h]), sc[m][h][0], sc[m][h][1], mn_lo, mn_hi);
                }
#pragma unroll 1                                                // unrolled it needs more than the 128 registers two CTAs leave
            for (int j = 0; j < 4; j++) {
                uint32_t lo[2][4], hi[2][4];
                int w0[2][2], w1[2][2];
#pragma unroll
                for (int m = 0; m < 2; m++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint2 w = ld<uint2>(p[m][h] + QS + 32 * j + 8 * t);
                        lo[m][h] = w.x & LO; lo[m][2 + h] = w.y & LO;
                        hi[m][h] = (w.x >> 4) & LO; hi[m][2 + h] = (w.y >> 4) & LO;
                        if (FMT == 5) {
                            constexpr uint32_t H4 = 0x10101010u;
                            const uint2 qh = ld<uint2>(p[m][h] + 16 + 8 * t);
                            const uint32_t x = __funnelshift_l(qh.x, qh.x, 4 - 2 * j), y = __funnelshift_l(qh.y, qh.y, 4 - 2 * j);   // bit 2 j of each byte to bit 4
                            lo[m][h] |= x & H4; lo[m][2 + h] |= y & H4;
                            hi[m][h] |= (x >> 1) & H4; hi[m][2 + h] |= (y >> 1) & H4;
                        }
                        w0[m][h] = (int)(sc[m][h][0] & 0xffu); w1[m][h] = (int)((sc[m][h][0] >> 8) & 0xffu);
                        sc[m][h][0] = __funnelshift_r(sc[m][h][0], sc[m][h][1], 16); sc[m][h][1] >>= 16;
                    }
#pragma unroll
                for (int n = 0; n < NTW; n++) {
                    const uint2 xl = ld<uint2>(xa + n * 8 * B::XP + 64 * j + 8 * t), xh = ld<uint2>(xa + n * 8 * B::XP + 64 * j + 32 + 8 * t);
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        int c0[4], c1[4];
                        mma0_u8s8_k32(c0, lo[m], xl.x, xl.y);
                        mma0_u8s8_k32(c1, hi[m], xh.x, xh.y);
#pragma unroll
                        for (int i = 0; i < 4; i++) tot[m][n][i] += w0[m][i >> 1] * c0[i] + w1[m][i >> 1] * c1[i];
                    }
                }
            }
#pragma unroll
            for (int m = 0; m < 2; m++) {
                const uint4 hA = ld<uint4>(p[m][0]), hB = ld<uint4>(p[m][1]);
                uint32_t u0, u1, mA[2], mB[2];
                k4_unpack(hA, u0, u1, mA[0], mA[1]);
                k4_unpack(hB, u0, u1, mB[0], mB[1]);
                const uint32_t a0 = t == 0 ? mA[0] : t == 1 ? mA[1] : 0u, a1 = t == 0 ? mB[0] : t == 1 ? mB[1] : 0u;
                const float2 fA = __half22float2(*reinterpret_cast<const __half2*>(&hA.x)), fB = __half22float2(*reinterpret_cast<const __half2*>(&hB.x));
#pragma unroll
                for (int n = 0; n < NTW; n++) {
                    const uint32_t bl = t < 2 ? ld<uint32_t>(dg + n * 8 * B::DG + 4 * t) : 0u, bh = t < 2 ? ld<uint32_t>(dg + n * 8 * B::DG + 8 + 4 * t) : 0u;
                    const float2 d8 = ld<float2>(sp + St::D + (wn * NTW * 8 + n * 8 + 2 * t) * 4);
                    const float e0 = d8.x, e1 = d8.y;
                    int sm[4];
                    mma0_u8s8_k16(sm, a0, a1, bh);
#pragma unroll
                    for (int i = 0; i < 4; i++) sm[i] <<= 6;
                    mma_u8s8_k16(sm, a0, a1, bl);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float2 f = i >> 1 ? fB : fA;
                        const float e = i & 1 ? e1 : e0;
                        acc[m][n][i] += (f.x * e) * (float)tot[m][n][i] - (f.y * e) * (float)sm[i];
                    }
                }
            }
        } else {
            constexpr uint32_t LO = 0x0f0f0f0fu, H2 = 0x30303030u;
#pragma unroll 1
            for (int n2 = 0; n2 < 2; n2++)
#pragma unroll 1
                for (int i2 = 0; i2 < 2; i2++) {
                    uint32_t q[2][2][4], sc[2][2][2];     // [tile][row half][quadrant]; scales of quadrants 0, 1 / 2, 3 in bytes 0 and 2
                    const uint32_t o = 16 * i2 + 4 * t;
#pragma unroll
                    for (int m = 0; m < 2; m++)
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const uint8_t* const b = p[m][h];
                            const uint32_t l0 = ld_u2(b + 64 * n2 + o), l1 = ld_u2(b + 64 * n2 + 32 + o), hb = ld_u2(b + 128 + 32 * n2 + o);
                            q[m][h][0] = (l0 & LO) | ((hb << 4) & H2); q[m][h][1] = (l1 & LO) | ((hb << 2) & H2);
                            q[m][h][2] = ((l0 >> 4) & LO) | (hb & H2); q[m][h][3] = ((l1 >> 4) & LO) | ((hb >> 2) & H2);
                            sc[m][h][0] = ld_u2(b + 192 + 8 * n2) >> (8 * i2);
                            sc[m][h][1] = ld_u2(b + 196 + 8 * n2) >> (8 * i2);
                        }
#pragma unroll
                    for (int z = 0; z < 4; z++)
#pragma unroll
                        for (int n = 0; n < NTW; n++) {
                            const uint32_t bx = ld<uint32_t>(xa + n * 8 * B::XP + 128 * n2 + 32 * z + 16 * i2 + 4 * t);
#pragma unroll
                            for (int m = 0; m < 2; m++) {
                                int c[4];
                                mma0_u8s8_k16(c, q[m][0][z], q[m][1][z], bx);
#pragma unroll
                                for (int i = 0; i < 4; i++) tot[m][n][i] += (int)(int8_t)((sc[m][i >> 1][z >> 1] >> (16 * (z & 1))) & 0xffu) * c[i];
                            }
                        }
                }
            uint32_t as[2][2];
            float d[2][2];
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int h = 0; h < 2; h++) { as[m][h] = ld_u2(p[m][h] + 192 + 4 * t); d[m][h] = f16_bits_to_f32(ld<uint16_t>(p[m][h] + 208)); }
#pragma unroll
            for (int n = 0; n < NTW; n++) {
                const uint32_t bl = ld<uint32_t>(dg + n * 8 * B::DG + 4 * t), bh = ld<uint32_t>(dg + n * 8 * B::DG + 16 + 4 * t);
                const float2 d8 = ld<float2>(sp + St::D + (wn * NTW * 8 + n * 8 + 2 * t) * 4);
                const float e0 = d8.x, e1 = d8.y;
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    int bias[4] = {0, 0, 0, 0};
                    mma_s8s8_k16(bias, as[m][0], as[m][1], bh);
#pragma unroll
                    for (int i = 0; i < 4; i++) bias[i] <<= 6;
                    mma_s8s8_k16(bias, as[m][0], as[m][1], bl);
#pragma unroll
                    for (int i = 0; i < 4; i++) acc[m][n][i] += (d[m][i >> 1] * (i & 1 ? e1 : e0)) * (float)(tot[m][n][i] - 32 * bias[i]);
                }
            }
        }
    }

    auto store = [&](uint32_t row, uint32_t tok, float v) {
        if (row >= seg_rows || tok >= a.batch) return;
        const size_t at = (size_t)tok * a.y_stride + a.y_off[s] + row;
        if (a.resid != nullptr) v = __fadd_rn(__ldcg(a.resid + at), v);
        a.y[at] = v;
    };
    if (KS == 1) {
#pragma unroll
        for (int n = 0; n < NTW; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t tok = tok0 + (wn * NTW + n) * 8 + 2 * t + (i & 1), rr = g + 8 * (i >> 1);
                if (SW) {
                    store(r0 + wm * 16 + rr, tok, silu_ref(acc[0][n][i]) * acc[1][n][i]);
                } else {
#pragma unroll
                    for (int m = 0; m < 2; m++) store(r0 + wm * 32 + m * 16 + rr, tok, acc[m][n][i]);
                }
            }
        return;
    }
    // every CTA leaves its part [token][rows] in shared memory; the outputs are dealt to the CTAs, parts added in rank order
    __syncthreads();
    float* part = reinterpret_cast<float*>(smem);
    constexpr uint32_t PP = G_ROWS + 1;
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int n = 0; n < NTW; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) part[((wn * NTW + n) * 8 + 2 * t + (i & 1)) * PP + wm * 32 + m * 16 + g + 8 * (i >> 1)] = acc[m][n][i];
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    auto total_at = [&](uint32_t v, uint32_t r) {
        const uint32_t at = ring + (v * PP + r) * 4;
        float f = 0.0f;
        for (uint32_t q = 0; q < KS; q++) {
            uint32_t remote;
            float x;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(q));
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(remote) : "memory");
            f = q ? f + x : x;
        }
        return f;
    };
    constexpr uint32_t OUT = SW ? G_ROWS / 2 : G_ROWS;      // output rows of the tile
    for (uint32_t i = rank * G_THREADS + tid; i < N * OUT; i += KS * G_THREADS) {
        const uint32_t v = i / OUT, r = i % OUT;
        if (SW) {
            const uint32_t at = (r >> 4) * 32 + (r & 15u);
            store(r0 + r, tok0 + v, silu_ref(total_at(v, at)) * total_at(v, at + 16));
        } else {
            store(r0 + r, tok0 + v, total_at(v, r));
        }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int FMT, int WM, int WN, int NTW, bool SW>
int launch_one(KqGemmArgs a, const LaunchCfg& cfg) {
    static bool done[64] = {};
    using St = KqStage<FMT, WM, WN, NTW>;
    auto kern = kq_gemm_kernel<FMT, WM, WN, NTW, SW>;
    a.stages = 3 * St::BYTES <= 112 * 1024 ? 3 : 2;
    const size_t smem = (size_t)a.stages * St::BYTES;
    static_assert(2 * St::BYTES <= 112 * 1024, "two CTAs an SM");
    static_assert(2 * St::BYTES >= St::N * (St::ROWS + 1) * 4, "the parts of a split reuse the stages");
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return ALICE_E_CUDA;
    if (dev >= 64 || !done[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return ALICE_E_CUDA;
        if (dev < 64) done[dev] = true;
    }
    constexpr uint32_t per = SW ? St::ROWS / 2 : St::ROWS;
    for (uint32_t i = 0; i < a.nw; i++) a.tile0[i + 1] = a.tile0[i] + (a.rows[i] + per - 1) / per;
    const uint32_t tiles = a.tile0[a.nw], toks = (a.batch + St::N - 1) / St::N, slots = 2 * (uint32_t)std::max(cfg.num_sms, 1);
    // columns shared by a cluster while that fills the two CTAs an SM holds and leaves each at least four blocks
    uint32_t KS = 1;
    while (KS < 8 && tiles * toks * KS * 2 <= slots && a.nb >= 8 * KS) KS *= 2;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(tiles * KS, toks); lc.blockDim = dim3(St::THREADS); lc.dynamicSmemBytes = smem; lc.stream = cfg.stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = KS; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = KS > 1 ? at : at + 1;
    lc.numAttrs = (KS > 1 ? 1 : 0) + (cfg.pdl ? 1 : 0);
    return cudaLaunchKernelEx(&lc, kern, a, KS) == cudaSuccess ? ALICE_OK : ALICE_E_CUDA;
}
template <int FMT, bool SW>
int launch_n(const KqGemmArgs& a, const LaunchCfg& cfg) {
    if (a.batch <= 16) return launch_one<FMT, 4, 1, 2, SW>(a, cfg);
    if (a.batch <= 32) return launch_one<FMT, 4, 1, 4, SW>(a, cfg);
    return launch_one<FMT, 2, 2, 4, SW>(a, cfg);      // in tiles of 64 also what the tcgen05 kernel could not take (no tensor map, no scratch)
}
template <int FMT>
int launch_fmt(const KqGemmArgs& a, const LaunchCfg& cfg) { return a.up ? launch_n<FMT, true>(a, cfg) : launch_n<FMT, false>(a, cfg); }

}  // namespace

int launch_kq_gemm(const GemvOp& op, const LaunchCfg& cfg) {
    const WeightDesc& w0 = *op.w[0];
    const bool q4 = w0.fmt == WF_Q4_K, q5 = w0.fmt == WF_Q5_K;
    if ((!q4 && !q5 && w0.fmt != WF_Q6_K) || !op.q8 || op.argmax_key || op.npeers || op.norm_w) return ALICE_E_SHAPE;
    if (op.nw < 1 || op.nw > 3 || (op.up && op.nw != 1) || w0.cols % 256 || op.q8->nb * 256 != w0.cols) return ALICE_E_SHAPE;
    if (((uintptr_t)op.q8->qs & 15) || ((uintptr_t)op.q8->bsums & 15) || !op.y) return ALICE_E_SHAPE;
    KqGemmArgs a = {};
    uint32_t total = 0;
    for (uint32_t i = 0; i < op.nw; i++) {
        const WeightDesc* w = op.w[i];
        if (!w || !w->rows || !w->data || ((uintptr_t)w->data & 15) || w->fmt != w0.fmt || w->cols != w0.cols || w->row_bytes != w0.row_bytes) return ALICE_E_SHAPE;
        a.w[i] = w->data; a.rows[i] = w->rows; a.y_off[i] = op.y_off[i];
        total += w->rows;
    }
    if (op.up) {
        const WeightDesc& u = *op.up;
        if (u.fmt != w0.fmt || u.rows != w0.rows || u.cols != w0.cols || u.row_bytes != w0.row_bytes || !u.data || ((uintptr_t)u.data & 15)) return ALICE_E_SHAPE;
        a.up = u.data;
    }
    if (op.batch > 64) {
        const int rc = launch_kq_gemm_tc(op, cfg);
        if (rc != ALICE_E_SHAPE) return rc;
    }
    a.nw = op.nw; a.row_bytes = w0.row_bytes; a.nb = w0.cols / 256;
    a.qs = op.q8->qs; a.d = op.q8->d; a.bsums = op.q8->bsums;
    a.y = op.y; a.resid = op.resid; a.y_stride = op.y_stride ? op.y_stride : total; a.batch = op.batch;
    return q4 ? launch_fmt<4>(a, cfg) : q5 ? launch_fmt<5>(a, cfg) : launch_fmt<6>(a, cfg);
}

}  // namespace alice

// K-quant products with more than 64 vectors on the fifth-generation tensor cores (tcgen05.mma kind::f16).
//
// A weight enters as the integer scale x quant, an activation as its Q8_K integer, both exact in f16: up to 63 * 31 for Q4_K / Q5_K;
// for Q6_K (up to 128 * 32) the scale as a multiple of 16 and -8 .. 7, two products. The f32 accumulator of one 256-column block then holds
// the integer dot of q4k_q8k_dot / q6k_q8k_dot (src/gguf.rs:3201-3251, :3282-3319), a second one the min term (sums of 16 activations,
// at most 2048, times the 6-bit mins), and both are scaled by the block's f16 and f32 factors and added up in f32 registers once per block.
//
// The dot is exact up to 2^24; weights of an ordinary matrix and activations of both signs give some 3e5. Activations of one sign, all near
// the largest of their block, can pass it (Q5_K reaches 3.8 times 2^24, Q6_K 8 times); every step of 16 columns beyond it then rounds by
// less than 2^-23 of the sum. Measured on such blocks: 4 to 11 * 2^-24 of a result, 0.6 to 1.2 by integer sums. Draining before 2^24 (every 128
// or 64 columns) is exact there, but adds a block up in pieces, which costs bits on ordinary blocks (error of a row of 56 blocks 2.0e-7 for
// two pieces, 2.8e-7 for four, 1.5e-7 for one, 1.6e-7 by integer sums) and a tenth of the time of a prompt.
//
// One CTA per SM, 128 rows x 128 vectors, 20 warps: 8 unpack raw blocks (cp.async, a block ahead) into the swizzled A tiles, half a row a
// thread, one warp copies the B tiles by TMA, one issues the products, 8 drain the accumulators of the block before (two sets in TMEM), 16 vectors
// ahead, which takes registers the other warps give up (72 and 48 against 144). Where tiles are fewer than the SMs a cluster shares the
// columns and adds its parts through distributed shared memory in rank order.
// Gate and up of an 8B model with 256 vectors, step by step: 216 us with four unpacking warps, 162 with eight, 140 with the tiles over whole waves split by
// columns (launch_tc), 128 with the registers moved and 16 vectors at a time (137 with 96 registers for all and 8), 122 with two k-tiles to a hand-over (Q4_K; the
// shallower rings of the others lose by it, Q5_K 152 and 164). Q6_K reads its words for two k-tiles at a time and multiplies by the two parts of the
// scale: 4096 x 14336 with 256 vectors 126 -> 102 us. Waits by one lane of a warp, or a row a thread and every other k-tile, are no faster (150, 132 us).
// What bounds it: the hand-overs. No unit is near its peak (ALU 34 %, tensor pipe 28, shared memory 45, issue slots 57), and without unpacking and
// draining 104 of the 128 us were left. A 256-token prompt of an 8B model takes 12.2 ms, 23.0 by the integer path of mma.sync (csrc/gemm_kq.cu), which
// spends some 16 instructions per product on scales and unpacking.
#include <algorithm>

#include "../../include/alice_cuda.h"
#include "common.cuh"
#include "gemm_kq.cuh"
#include "gemv_kq_mma.cuh"
#include "tc_dev.cuh"

namespace alice {
namespace {

constexpr uint32_t KT_M = 128, KT_N = 128, KT_PROD = 256, KT_EPI = 256, KT_THREADS = KT_PROD + KT_EPI + 128;
constexpr uint32_t KT_R = 96, KT_RU = 72, KT_RD = 144, KT_RM = 48;      // registers a thread at launch, then of the unpacking, draining and other warps
static_assert(KT_PROD * KT_RU + KT_EPI * KT_RD + 128 * KT_RM <= KT_THREADS * KT_R, "a warpgroup would wait for registers for good");
constexpr int KERR_KT_WAIT = 7;      // as the bf16 product: operands or accumulators of a tensor-core product

template <int FMT> struct KtFmt;     // bytes of a raw block, 16-byte pieces and pitch of a raw row, k-tiles of a block, A tiles, ring depth, k-tiles unpacked at once
template <> struct KtFmt<4> { static constexpr uint32_t BB = 144, CH = 9, PITCH = 144, TILES = 5, ASUB = 1, STAGES = 5, PER = 2; };
template <> struct KtFmt<5> { static constexpr uint32_t BB = 176, CH = 11, PITCH = 176, TILES = 5, ASUB = 1, STAGES = 4, PER = 1; };
template <> struct KtFmt<6> { static constexpr uint32_t BB = 210, CH = 14, PITCH = 240, TILES = 4, ASUB = 2, STAGES = 3, PER = 1; };

template <int FMT>
struct KtGeom {
    using F = KtFmt<FMT>;
    static constexpr uint32_t A = 16384 * F::ASUB, STAGE = A + 16384, RAW = KT_M * F::PITCH, RING = F::STAGES * STAGE, SMEM = 1024 + RING + 2 * RAW,
                              KB = F::TILES * 64;      // columns of the prepared activations per block
    static_assert(RING >= KT_N * (KT_M + 1) * 4, "the parts of the result reuse the ring");
    static_assert(SMEM <= 226 * 1024, "shared memory of a CTA");
};

struct KtArgs {
    const uint8_t* w[3];
    uint32_t rows[3], y_off[3], tile0[4], nw;
    const uint8_t* up;
    uint32_t row_bytes, nb, dstride;
    const float* dt;             // [nb][dstride]: Q8_K scales
    float* y;
    const float* resid;
    uint32_t y_stride, batch, tile_lo;      // tile_lo: first tile of the launch
    int* status;
    CUtensorMap tb;
};

// Activations as the B tiles want them: x[v][blk * KB + ...] in f16, the columns in the order the unpacked weights have (Q4_K / Q5_K: second
// and third of every four exchanged), behind a Q4_K / Q5_K block its 16 sums and zeros; scales transposed (what lies there for vectors
// past the batch reaches their results only, which are not stored).
template <int FMT>
__global__ void __launch_bounds__(256) kt_prepare_kernel(const int8_t* qs, const float* d, const int16_t* bsums, uint32_t batch, uint32_t nb, uint32_t dstride, __half* x, float* dt) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr uint32_t KB = KtGeom<FMT>::KB;
    const uint32_t lane = threadIdx.x & 31, i = blockIdx.x * 8 + (threadIdx.x >> 5);     // a warp per block
    if (i >= batch * nb) return;
    const uint32_t v = i / nb, b = i - v * nb;
    __half* out = x + ((size_t)v * nb + b) * KB;
    const uint2 q = __ldcg(reinterpret_cast<const uint2*>(qs + (size_t)i * 256) + lane);
    uint32_t h[4];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const uint32_t w = k ? q.y : q.x;
        __half e[4];
#pragma unroll
        for (int j = 0; j < 4; j++) e[j] = __int2half_rn((int)(int8_t)(w >> (8 * j)));
        const __half2 p0 = FMT == 6 ? __halves2half2(e[0], e[1]) : __halves2half2(e[0], e[2]), p1 = FMT == 6 ? __halves2half2(e[2], e[3]) : __halves2half2(e[1], e[3]);
        h[2 * k] = *reinterpret_cast<const uint32_t*>(&p0);
        h[2 * k + 1] = *reinterpret_cast<const uint32_t*>(&p1);
    }
    reinterpret_cast<uint4*>(out)[lane] = make_uint4(h[0], h[1], h[2], h[3]);
    if (FMT != 6) {
        const __half2 z = __half2half2(__ushort_as_half(0));
        const __half2 s = lane < 8 ? __halves2half2(__int2half_rn(bsums[(size_t)i * 16 + 2 * lane]), __int2half_rn(bsums[(size_t)i * 16 + 2 * lane + 1])) : z;
        reinterpret_cast<__half2*>(out + 256)[lane] = s;
    }
    if (lane == 0) dt[(size_t)b * dstride + v] = __ldcg(d + i);
}

__device__ __forceinline__ uint32_t h2u(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }
__device__ __forceinline__ __half2 u2h(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
template <class V> __device__ __forceinline__ V kld(const uint8_t* p) { return *reinterpret_cast<const V*>(p); }
__device__ __forceinline__ uint32_t kld_u2(const uint8_t* p) {      // a 32-bit word at a 2-byte boundary
    const uint32_t a = smem_u32(p) & 2u;
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p - a);
    return __funnelshift_r(q[0], q[1], a * 8u);
}

// `scales`: those of the block half's sub-blocks, this thread's in bytes 0 and 2.
// 32 weights (k-half `half` of k-tile c) of a raw block as f16 integers into logical 16-byte pieces 4 half .. of row r of the A tile at `at`.
template <int FMT>
__device__ __forceinline__ void kt_unpack(const uint8_t* raw, uint32_t scales, uint32_t c, uint32_t half, uint8_t* at, uint32_t r) {
    if constexpr (FMT != 6) {
        const uint32_t j = 2 * c + half, sc = (scales >> (16 * (c & 1))) & 0xffu;
        // a high nibble stays where it is in its byte: 1024 + 16 quant, times scale / 16
        const __half2 one = __half2half2(__ushort2half_rn((unsigned short)sc)), s2 = half ? __hmul2(one, __float2half2_rn(0.0625f)) : one;
        const __half2 o2 = __hmul2(s2, __float2half2_rn(-1024.0f));
        const uint32_t mask = half ? 0x00f000f0u : 0x000f000fu;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const uint4 q4 = kld<uint4>(raw + (FMT == 5 ? 48 : 16) + 32 * c + 16 * i);
            const uint32_t w[4] = {q4.x, q4.y, q4.z, q4.w};
            uint32_t hb[4] = {0u, 0u, 0u, 0u};
            if (FMT == 5) {
                const uint4 h4 = kld<uint4>(raw + 16 + 16 * i);
                hb[0] = h4.x >> j; hb[1] = h4.y >> j; hb[2] = h4.z >> j; hb[3] = h4.w >> j;
            }
            uint32_t out[8];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                uint32_t e = (w[k] & mask) | 0x64006400u, o = ((w[k] >> 8) & mask) | 0x64006400u;
                if (FMT == 5) {
                    const uint32_t up = half ? 8 : 4;
                    e |= (hb[k] & 0x00010001u) << up; o |= ((hb[k] >> 8) & 0x00010001u) << up;
                }
                out[2 * k] = h2u(__hfma2(u2h(e), s2, o2));
                out[2 * k + 1] = h2u(__hfma2(u2h(o), s2, o2));
            }
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const uint32_t piece = 4 * half + 2 * i + k;
                *reinterpret_cast<uint4*>(at + r * 128 + ((piece ^ (r & 7u)) * 16)) = make_uint4(out[4 * k], out[4 * k + 1], out[4 * k + 2], out[4 * k + 3]);
            }
        }
    }
}
// Q6_K: the words with the quants of k-tiles c and c + 1 (c even), word w = (k + r / 8) % 4 of either 16 columns: rows eight apart meet the same banks.
__device__ __forceinline__ void k6_load(const uint8_t* raw, uint32_t c, uint32_t half, uint32_t rot, uint32_t (&l)[8], uint32_t (&h)[8]) {
    const uint8_t* ql = raw + 32 * c + 32 * half;
    const uint8_t* qh = raw + 128 + 16 * c;
#pragma unroll
    for (uint32_t j = 0; j < 8; j++) {
        const uint32_t at = 16 * (j >> 2) + 4 * ((j + rot) & 3u);
        l[j] = kld_u2(ql + at);
        h[j] = kld_u2(qh + at);
    }
}
// 32 weights (k-half `half` of k-tile c) into row r of the two A tiles at `at`: quant times a multiple of 16 next to the scale, and times the rest.
__device__ __forceinline__ void k6_unpack(const uint8_t* raw, const uint32_t (&l)[8], const uint32_t (&h)[8], uint32_t c, uint32_t half, uint32_t rot, uint8_t* at, uint32_t r) {
    const uint32_t z = 2 * (c & 1) + half;                    // quadrant of half c / 2 of the block
    uint8_t* const row = at + r * 128;
    const uint32_t base = (4 * half ^ (r & 7u)) << 4;
#pragma unroll
    for (uint32_t i = 0; i < 2; i++) {
        const int sc = (int)(int8_t)raw[192 + 8 * (c >> 1) + 2 * z + i], up = (sc + 8) & ~15;
        const __half2 s_hi = __half2half2(__int2half_rn(up)), s_lo = __half2half2(__int2half_rn(sc - up));
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {
            const uint32_t w = (k + rot) & 3u, j = 4 * i + k;
            const uint32_t lw = c & 1 ? l[j] >> 4 : l[j];
            const uint32_t hx = c & 1 ? h[j] >> (2 * half) : (half ? h[j] << 2 : h[j] << 4);
            const uint32_t q = ((lw & 0x0f0f0f0fu) | (hx & 0xf0f0f0f0u)) & 0x3f3f3f3fu;
            uint32_t hi[2], lo[2];
#pragma unroll
            for (int p = 0; p < 2; p++) {                     // bytes 2 p and 2 p + 1, in order
                const __half2 u = __hsub2(u2h(__byte_perm(q, 0x64u, p ? 0x4342u : 0x4140u)), __float2half2_rn(1056.0f));      // quant - 32
                hi[p] = h2u(__hmul2(u, s_hi));
                lo[p] = h2u(__hmul2(u, s_lo));
            }
            const uint32_t to = base ^ (i << 5) ^ (w << 3);
            *reinterpret_cast<uint2*>(row + to) = make_uint2(hi[0], hi[1]);
            *reinterpret_cast<uint2*>(row + 16384 + to) = make_uint2(lo[0], lo[1]);
        }
    }
}
// The mins of a Q4_K / Q5_K block, each for two sums of 16: pieces 0 and 1 of the row.
__device__ __forceinline__ void kt_mins(uint32_t m, uint32_t half, uint8_t* at, uint32_t r) {
    uint32_t out[4];
#pragma unroll
    for (int k = 0; k < 4; k++) out[k] = h2u(__half2half2(__ushort2half_rn((unsigned short)((m >> (8 * k)) & 0xffu))));
    *reinterpret_cast<uint4*>(at + r * 128 + ((half ^ (r & 7u)) * 16)) = make_uint4(out[0], out[1], out[2], out[3]);
}

template <uint32_t N> __device__ __forceinline__ void regs_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <uint32_t N> __device__ __forceinline__ void regs_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

template <int FMT, bool SW>
__global__ void __launch_bounds__(KT_THREADS, 1) kq_gemm_tc_kernel(const __grid_constant__ KtArgs a, const uint32_t KS) {
    using F = KtFmt<FMT>;
    using G = KtGeom<FMT>;
    extern __shared__ uint8_t raw_smem[];
    __shared__ __align__(8) uint64_t full_[F::STAGES], empty_[F::STAGES], tfull_[2], tempty_[2], drain_;
    __shared__ uint32_t tmem_base;
    // Q8_K scales of the vectors, four blocks deep: when the copies of block k are asked for, block k - 3 has been drained
    __shared__ __align__(16) float dts[4][KT_N];
    uint8_t* const ring = raw_smem + (1024u - (smem_u32(raw_smem) & 1023u));
    uint8_t* const raw = ring + G::RING;
    const uint32_t ring_s = smem_u32(ring);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    auto bar = [](uint64_t* b, uint32_t i) { return smem_u32(b + i); };
    const uint32_t rank = KS > 1 ? blockIdx.x % KS : 0u, tile = a.tile_lo + blockIdx.x / KS, tok0 = blockIdx.y * KT_N;
    uint32_t s = 0;
    if (!SW) while (s + 1 < a.nw && tile >= a.tile0[s + 1]) s++;
    constexpr uint32_t OUT = SW ? KT_M / 2 : KT_M;
    const uint32_t seg_rows = a.rows[s], r0 = (tile - a.tile0[s]) * OUT;
    const uint32_t b_lo = a.nb * rank / KS, nblk = a.nb * (rank + 1) / KS - b_lo;
    pdl_launch_dependents();
    if (tid == 0) {
        for (uint32_t i = 0; i < F::STAGES; i++) { mbar_init(bar(full_, i), KT_PROD + 1); mbar_init(bar(empty_, i), 1); }
        for (uint32_t i = 0; i < 2; i++) { mbar_init(bar(tfull_, i), 1); mbar_init(bar(tempty_, i), KT_EPI); }
        mbar_init(smem_u32(&drain_), 1);
        mbar_fence_init();
        fence_proxy_async();
    }
    if (warp == 17) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "n"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    // row of the matrix behind row i of the tile: with SwiGLU 64 gate rows, then the same 64 of up
    auto matrix = [&](uint32_t i) { return SW && i >= KT_M / 2 ? a.up : a.w[s]; };
    auto matrix_row = [&](uint32_t i) { return min(r0 + (SW ? i & (KT_M / 2 - 1) : i), seg_rows - 1); };
    float* const part = reinterpret_cast<float*>(ring);            // [vector][128 rows]
    constexpr uint32_t PP = KT_M + 1;
    bool ok = true;

    if (warp < 8) {                       // ---- unpack
        regs_down<KT_RU>();
        const uint32_t r = tid >> 1, half = tid & 1u;
        const uint64_t total = (uint64_t)seg_rows * a.row_bytes;
        auto fetch = [&](uint32_t k) {
            if (k < nblk) {
                uint8_t* const dst = raw + (k & 1u) * G::RAW;
#pragma unroll 2
                for (uint32_t i = tid; i < KT_M * F::CH; i += KT_PROD) {
                    const uint32_t row = i / F::CH, c = i - row * F::CH;
                    const uint64_t off = (((uint64_t)matrix_row(row) * a.row_bytes + (uint64_t)(b_lo + k) * F::BB) & ~(uint64_t)15) + c * 16;
                    const uint32_t n = off < total ? (uint32_t)min((uint64_t)16, total - off) : 0u;
                    const uint8_t* m = matrix(row);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + row * F::PITCH + c * 16)), "l"(n ? m + off : m), "r"(n) : "memory");
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        fetch(0);                         // weights: nothing of the kernel ahead
        uint32_t it = 0;
        for (uint32_t k = 0; k < nblk; k++) {      // a warp whose wait ran out still meets the others at the barriers
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            asm volatile("bar.sync 1, %0;" ::"n"(KT_PROD) : "memory");          // block k is in, everyone is done with block k - 1
            fetch(k + 1);
            const uint8_t* src = raw + (k & 1u) * G::RAW + r * F::PITCH;
            if (FMT == 6) src += (matrix_row(r) * a.row_bytes + (b_lo + k) * F::BB) & 15u;
            uint32_t sl = 0, sh = 0, ml = 0, mh = 0, ql[8], qh[8];
            const uint32_t rot = r >> 3;
            if (FMT != 6) k4_unpack(kld<uint4>(src), sl, sh, ml, mh);
#pragma unroll
            for (uint32_t c0 = 0; c0 + F::PER <= F::TILES; c0 += F::PER) {
                const uint32_t n = c0 + 2 * F::PER > F::TILES ? F::TILES - c0 : F::PER;      // the last takes the rest along
#pragma unroll
                for (uint32_t j = 0; j < n; j++) ok = ok && mbar_wait(bar(empty_, (it + j) % F::STAGES), (((it + j) / F::STAGES) & 1) ^ 1);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
#pragma unroll
                for (uint32_t j = 0; j < n; j++) {
                    const uint32_t c = c0 + j;
                    uint8_t* const at = ring + (it + j) % F::STAGES * G::STAGE;
                    if constexpr (FMT == 6) {
                        if (!(c & 1)) k6_load(src, c, half, rot, ql, qh);
                        k6_unpack(src, ql, qh, c, half, rot, at, r);
                    } else if (c == 4) {
                        kt_mins(half ? mh : ml, half, at, r);
                    } else {
                        kt_unpack<FMT>(src, half ? (c < 2 ? sl >> 8 : sh >> 8) : (c < 2 ? sl : sh), c, half, at, r);
                    }
                }
                fence_proxy_async();
#pragma unroll
                for (uint32_t j = 0; j < n; j++) mbar_arrive(bar(full_, (it + j) % F::STAGES));
                it += n;
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();                  // the ring is free: all products and copies are done
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        regs_up<KT_R>();
    } else if (warp < 16) {               // ---- drain
        regs_up<KT_RD>();
        float acc[64];
        const uint32_t quad = warp & 3u, ch = (warp - 8) >> 2, i = quad * 32 + lane;
        const uint8_t* wrow = matrix(i) + (uint64_t)matrix_row(i) * a.row_bytes;
#pragma unroll
        for (int j = 0; j < 64; j++) acc[j] = 0.0f;
        pdl_wait();
        // scale (and min factor) of this row's block, a block ahead
        auto head = [&](uint32_t k) -> uint32_t {
            const uint8_t* blk = wrow + (uint64_t)(b_lo + min(k, nblk - 1)) * F::BB;
            return FMT == 6 ? (uint32_t)__ldg(reinterpret_cast<const unsigned short*>(blk + 208)) : __ldg(reinterpret_cast<const uint32_t*>(blk));
        };
        uint32_t hd = head(0);
        for (uint32_t k = 0; k < nblk; k++) {
            const uint32_t b = k & 1u;
            const float2 f = __half22float2(u2h(hd));
            hd = head(k + 1);
            ok = __all_sync(0xffffffffu, mbar_wait(bar(tfull_, b), (k >> 1) & 1));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t base = tmem + b * KT_N + ch * 64 + ((quad * 32) << 16);
            const float* e = dts[k & 3u] + ch * 64;
            uint32_t p[2][16], m[2][16];      // a piece of 16 vectors ahead
            tmem_get16(p[0], base);
            if (FMT != 6) tmem_get16(m[0], base + 256);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                if (FMT != 6) tmem_got16(p[c & 1], m[c & 1]); else tmem_got16(p[c & 1]);
                if (c < 3) {
                    tmem_get16(p[(c + 1) & 1], base + 16 * c + 16);
                    if (FMT != 6) tmem_get16(m[(c + 1) & 1], base + 256 + 16 * c + 16);
                }
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    const float4 x4 = *reinterpret_cast<const float4*>(e + 16 * c + j);
                    const float x[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        float& y = acc[16 * c + j + q];
                        if (FMT != 6) y = fmaf(x[q], fmaf(-f.y, __uint_as_float(m[c & 1][j + q]), f.x * __uint_as_float(p[c & 1][j + q])), y);
                        else y = fmaf(f.x * x[q], __uint_as_float(p[c & 1][j + q]), y);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(bar(tempty_, b));
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();                  // the ring is free: all products and copies are done
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 64; j++) part[(ch * 64 + j) * PP + i] = acc[j];
        regs_down<KT_R>();
    } else {
    regs_down<KT_RM>();
    if (warp == 16) {              // ---- B tiles
        if (lane == 0) {
            pdl_wait();
            uint32_t it = 0;
            for (uint32_t k = 0; k < nblk && ok; k++)
                for (uint32_t c = 0; c < F::TILES; c++, it++) {
                    const uint32_t st = it % F::STAGES;
                    ok = mbar_wait(bar(empty_, st), ((it / F::STAGES) & 1) ^ 1);
                    if (!ok) break;
                    mbar_arrive_expect_tx(bar(full_, st), c == 0 ? 16384 + KT_N * 4 : 16384);
                    if (c == 0) bulk_g2s(smem_u32(dts[k & 3u]), a.dt + (size_t)(b_lo + k) * a.dstride + tok0, KT_N * 4, bar(full_, st));
                    tma_2d(ring_s + st * G::STAGE + G::A, &a.tb, (int)((b_lo + k) * G::KB + c * 64), (int)tok0, bar(full_, st));
                }
            // every copy has landed before the CTA may leave
            const uint32_t last = it < F::STAGES ? it : F::STAGES;
            for (uint32_t j = it - last; j < it; j++) mbar_wait(bar(full_, j % F::STAGES), (j / F::STAGES) & 1);
        }
        __syncwarp();
    } else if (warp == 17) {                              // ---- products
        {
            constexpr uint32_t idesc = (1u << 4) | ((KT_N / 8) << 17) | ((KT_M / 16) << 24);      // f16 x f16 -> f32
            uint32_t it = 0;
            for (uint32_t k = 0; k < nblk && ok; k++) {
                const uint32_t b = k & 1u, d = tmem + b * KT_N;
                ok = __all_sync(0xffffffffu, mbar_wait(bar(tempty_, b), ((k >> 1) & 1) ^ 1));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (uint32_t c = 0; c < F::TILES; c++, it++) {
                    const uint32_t st = it % F::STAGES;
                    ok = __all_sync(0xffffffffu, mbar_wait(bar(full_, st), (it / F::STAGES) & 1));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t at = ring_s + st * G::STAGE;
                    const uint64_t db = smem_desc(at + G::A);
                    if (elect_lane()) {
                        if (FMT != 6 && c == 4) {
                            mma_f16(d + 256, smem_desc(at), db, idesc, false);
                        } else {
#pragma unroll
                            for (uint32_t z = 0; z < F::ASUB; z++) {
                                const uint64_t da = smem_desc(at + z * 16384);
#pragma unroll
                                for (int kk = 0; kk < 4; kk++) mma_f16(d, da + 2 * kk, db + 2 * kk, idesc, c > 0 || z > 0 || kk > 0);
                            }
                        }
                        mma_commit(bar(empty_, st));
                        if (c + 1 == F::TILES) mma_commit(bar(tfull_, b));
                    }
                    __syncwarp();
                }
            }
            if (elect_lane()) mma_commit(smem_u32(&drain_));
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&drain_), 0)) && ok;
        }
        __syncwarp();
    }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();                  // the ring is free: all products and copies are done
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        regs_up<KT_R>();
    }
    if (!ok && lane == 0) atomicCAS(a.status, 0, KERR_KT_WAIT);
    auto meet = [&]() {
        if (KS > 1) {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else {
            __syncthreads();
        }
    };
    meet();
    auto total_at = [&](uint32_t v, uint32_t i) {
        if (KS == 1) return part[v * PP + i];
        const uint32_t at = ring_s + (v * PP + i) * 4;
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
    pdl_wait();                           // the residual may be what an earlier kernel wrote (threads that have not waited yet)
    for (uint32_t i = rank * KT_THREADS + tid; i < KT_N * OUT; i += KS * KT_THREADS) {
        const uint32_t v = i / OUT, r = i % OUT, tok = tok0 + v, row = r0 + r;
        if (tok >= a.batch || row >= seg_rows) continue;
        float f = total_at(v, r);
        if (SW) f = silu_ref(f) * total_at(v, r + KT_M / 2);
        const size_t at = (size_t)tok * a.y_stride + a.y_off[s] + row;
        if (a.resid != nullptr) f = __fadd_rn(__ldcg(a.resid + at), f);
        a.y[at] = f;
    }
    meet();
    if (warp == 17) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512));
}

template <int FMT, bool SW>
int launch_tc(KtArgs a, const GemvOp& op, const LaunchCfg& cfg) {
    using G = KtGeom<FMT>;
    static bool done[64] = {};
    auto kern = kq_gemm_tc_kernel<FMT, SW>;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return ALICE_E_CUDA;
    if (dev >= 64 || !done[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::SMEM) != cudaSuccess) return ALICE_E_CUDA;
        if (dev < 64) done[dev] = true;
    }
    constexpr uint32_t per = SW ? KT_M / 2 : KT_M;
    for (uint32_t i = 0; i < a.nw; i++) a.tile0[i + 1] = a.tile0[i] + (a.rows[i] + per - 1) / per;
    const uint32_t toks = (a.batch + KT_N - 1) / KT_N;
    a.dstride = toks * KT_N;
    // scratch: prepared activations, then scales
    const size_t xbytes = (size_t)a.batch * a.nb * G::KB * 2, need = xbytes + (size_t)a.nb * a.dstride * 4;
    if (!op.prep || ((uintptr_t)op.prep & 15) || need > op.prep_bytes) return ALICE_E_SHAPE;
    auto* x = static_cast<__half*>(op.prep);
    auto* dt = reinterpret_cast<float*>(static_cast<uint8_t*>(op.prep) + xbytes);
    a.dt = dt;
    if (!encode_fn() || !tile_map(&a.tb, x, a.batch, a.nb * G::KB, a.nb * G::KB, KT_N)) return ALICE_E_SHAPE;
    cudaLaunchConfig_t lc = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    lc.stream = cfg.stream;
    lc.gridDim = dim3((a.batch * a.nb + 7) / 8); lc.blockDim = dim3(256);
    lc.attrs = at + 1; lc.numAttrs = cfg.pdl ? 1 : 0;
    if (cudaLaunchKernelEx(&lc, kt_prepare_kernel<FMT>, op.q8->qs, op.q8->d, op.q8->bsums, a.batch, a.nb, a.dstride, x, dt) != cudaSuccess) return ALICE_E_CUDA;
    const uint32_t tiles = a.tile0[a.nw], sms = (uint32_t)std::max(cfg.num_sms, 1);
    // CTAs that share the columns of each of n tiles, where these leave SMs idle
    auto shares = [&](uint32_t n, uint32_t least) { uint32_t k = 1; while (k < 8 && n * toks * k * 2 <= sms && a.nb >= least * k) k *= 2; return k; };
    // Tiles over whole waves of the SMs, up to half a wave of them, are a launch of its own ahead of the others, their columns shared by clusters: a CTA
    // takes its blocks and, in blocks, 1.5 for its start, 2.5 with a cluster's sum, the launch 2.5, so from a.nb = 7 on it is shorter than a wave. Measured
    // with 256 vectors, without and with: gate and up of an 8B model (448 CTAs on 148 SMs) 162 and 140 us (Q5_K 195 and 161), 9728 x 4096 81
    // and 53, 13312 x 4096 (60 CTAs over) 82 and 70, 10240 x 2048 48 and 35, 13312 x 2048 49 and 49. Shares of the main launch, eight blocks at least.
    uint32_t rest = tiles * toks > sms ? (tiles * toks % sms + toks - 1) / toks : 0u;
    if (rest && (rest * toks * 2 > sms || a.nb / shares(rest, 2) + 6 > a.nb)) rest = 0;
    auto launch = [&](uint32_t lo, uint32_t n, uint32_t ks) {
        a.tile_lo = lo;
        at[0].val.clusterDim.x = ks;
        lc.gridDim = dim3(n * ks, toks); lc.blockDim = dim3(KT_THREADS); lc.dynamicSmemBytes = G::SMEM;
        lc.attrs = ks > 1 ? at : at + 1;
        lc.numAttrs = (ks > 1 ? 1 : 0) + (cfg.pdl ? 1 : 0);
        return cudaLaunchKernelEx(&lc, kern, a, ks) == cudaSuccess ? ALICE_OK : ALICE_E_CUDA;
    };
    const int rc = rest ? launch(tiles - rest, rest, shares(rest, 2)) : ALICE_OK;
    return rc ? rc : launch(0, tiles - rest, shares(tiles - rest, 8));
}

}  // namespace

size_t kq_tc_prep_bytes(uint32_t cols, uint32_t batch) {
    const size_t nb = (cols + 255) / 256;
    return (size_t)batch * nb * 640 + nb * ((batch + 127) / 128 * 128) * 4;
}

int launch_kq_gemm_tc(const GemvOp& op, const LaunchCfg& cfg) {
    const WeightDesc& w0 = *op.w[0];
    KtArgs a = {};
    uint32_t total = 0;
    for (uint32_t i = 0; i < op.nw; i++) {
        a.w[i] = op.w[i]->data; a.rows[i] = op.w[i]->rows; a.y_off[i] = op.y_off[i];
        total += op.w[i]->rows;
    }
    if (op.up) a.up = op.up->data;
    a.nw = op.nw; a.row_bytes = w0.row_bytes; a.nb = w0.cols / 256;
    a.y = op.y; a.resid = op.resid; a.y_stride = op.y_stride ? op.y_stride : total; a.batch = op.batch; a.status = cfg.status;
    if (op.up) return w0.fmt == WF_Q4_K ? launch_tc<4, true>(a, op, cfg) : w0.fmt == WF_Q5_K ? launch_tc<5, true>(a, op, cfg) : launch_tc<6, true>(a, op, cfg);
    return w0.fmt == WF_Q4_K ? launch_tc<4, false>(a, op, cfg) : w0.fmt == WF_Q5_K ? launch_tc<5, false>(a, op, cfg) : launch_tc<6, false>(a, op, cfg);
}

}  // namespace alice

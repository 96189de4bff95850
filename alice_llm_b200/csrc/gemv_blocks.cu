// Kernels and launch of csrc/gemv_blocks.cuh.
//
// A block is an f16 scale and 32 int8 (Q8_0), 128 signs (Q1_0) or 128 two-bit slots (Q2_0); blocks are 2-byte aligned.
//
// Q1_0 and Q2_0 run on the int8 tensor path: the f32 activations become 31-bit fixed point (unit 2^-30 of a power of two above the
// largest) in four signed base-256 digits; the digits of two vectors fill the eight B columns. A operand: bytes & (1 << j), or the
// two bits of a slot at once (0 .. 3 times 4^q). A block's sum is an exact integer (two digits joined in 32 bits: at most 16 bytes x
// 255 x 128 x 257), the offset of the codes is taken off in integers too (2 S - T, S - T with T summed over the same digits), and one
// f32 multiply-add per block scales it.
//
// Q8_0 runs in f32 throughout: fixed point with one exponent for a vector would take the bits of its small elements, and with them the
// results of rows whose weights at the large ones are near zero. A weight d * q has 19 bits, so it is exact; a lane keeps four rows x
// four columns of a block in registers and uses them for every vector, whose elements come from shared memory.
//
// Every warp has a ring of its own in shared memory (16 rows x 8 blocks a stage, cp.async, no barrier between warps); the digit
// table (Q8_0: the vectors) of a CTA's columns stays in shared memory for the whole launch. A cluster of S CTAs shares the columns
// where the table fits no single CTA or a matrix has few rows; the (tile, stage) pairs of a CTA are dealt evenly to its warps and the
// parts of a tile are added in a fixed order.
//
// What bounds it: Q8_0 the instructions (16 weights a lane and block to unpack, scale and multiply with each vector; 151936 x 5120 196 us
// for one vector, 228 by the ring kernel; 32768 x 4096 44 us for two, 57 for four, 99 for eight, 34 for each by the ring kernel); Q1_0 and
// Q2_0 the ALU for one or two vectors (Q1_0, one vector: 32 masks among some 60 bit operations per 576 bytes, one every other clk and SM quarter;
// more warps an SM, 20 to 32, gain nothing: 102400 x 5120 in 29.2 us, 2.5 TB/s, 32.4 with the addresses of every copied piece made anew), the products (8 per 16 rows and block of Q1_0, 4 of Q2_0, for each pair of vectors) for more.
#include <algorithm>

#include "../../include/alice_cuda.h"
#include "digits_dev.cuh"
#include "gemv_blocks.cuh"
#include "gemv_mma.cuh"
#include "packed_f32.cuh"

namespace alice {
namespace {

constexpr int BLK_WARPS = 16;
constexpr uint32_t BLK_ITEM = 8;                 // blocks of a row a stage holds
constexpr uint32_t BLK_SMEM = 224 * 1024, BLK_HDR = 128;

template <int FMT> struct BlkFmt;                // bytes and elements of a block, digit (or f32) bytes per block and pair of vectors, row pitch of a stage
// pitch: 32-bit reads of 8 rows x 16 bytes, or of 4 rows x 32 bytes for Q8_0, fill the banks once (48 or 32 modulo 128)
template <> struct BlkFmt<0> { static constexpr uint32_t BB = 34, EL = 32, DIG = 256, PITCH = 288; static constexpr bool T = false; };
template <> struct BlkFmt<1> { static constexpr uint32_t BB = 18, EL = 128, DIG = 1024, PITCH = 176; static constexpr bool T = true; };
template <> struct BlkFmt<2> { static constexpr uint32_t BB = 34, EL = 128, DIG = 1024, PITCH = 304; static constexpr bool T = true; };

struct BlkArgs {
    const uint8_t* w[3];
    uint32_t rows[3], y_off[3], tile0[4], nw;
    const uint8_t* up;
    uint32_t row_bytes, nb;                      // blocks of a row
    const float* x;                              // one or two vectors: the kernel makes the digits itself; more: the table. Q8_0: always
    const uint8_t* digits;                       // [nb][NT][DIG]
    const int* tsum;                             // [nb][NT][4]
    const float* kappa;
    float* y;
    const float* resid;
    uint32_t y_stride, batch;
    unsigned long long* argmax_key;
    uint32_t tiles_max, stages, tsum_off, main_off, head_off;      // shared memory: header | rings | digits | tsum | main | head
    int* status;
    long long wait_limit;
};

constexpr int BLK_FIX_BITS = 30;
// four signed base-256 digits of f, |f| <= 2^30, most significant first
__device__ __forceinline__ void block_digits(int f, int (&d)[4]) {
    d[3] = (int)(int8_t)(f & 255); f = (f - d[3]) >> 8;
    d[2] = (int)(int8_t)(f & 255); f = (f - d[2]) >> 8;
    d[1] = (int)(int8_t)(f & 255); f = (f - d[1]) >> 8;
    d[0] = f;
}

// Digits of one block by eight consecutive lanes (t = u & 3, h = u >> 2) into the block's record, columns 4 col .. + 3, and its two joined
// digit sums into tsum[0 .. 1]; `live` lanes store. FMT 1: byte 4 t + b, bits 4 h .. 4 h + 3; 2: byte
// 16 h + 4 t + b, its four slots.
template <int FMT>
__device__ __forceinline__ void block_record(const float* x, bool live, uint32_t u, uint32_t col, const FixedScale to_fixed, uint8_t* rec, int* tsum) {
    uint32_t out[4][4] = {};
    int ts[4] = {0, 0, 0, 0};
    const uint32_t t = u & 3u, h = u >> 2;
#pragma unroll
    for (uint32_t b = 0; b < 4; b++) {
        const uint32_t e = FMT == 1 ? 8 * (4 * t + b) + 4 * h : 4 * (16 * h + 4 * t + b);
        const float4 q = live ? __ldcg(reinterpret_cast<const float4*>(x + e)) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float xe[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (uint32_t jj = 0; jj < 4; jj++) {
            const int sh = FMT == 1 ? (int)(4 * h + jj) : (int)(2 * jj);
            const int f = (to_units(xe[jj], to_fixed) + ((1 << sh) >> 1)) >> sh;
            int dg[4];
            block_digits(f, dg);
#pragma unroll
            for (int d = 0; d < 4; d++) {
                out[d][jj] |= (uint32_t)(dg[d] & 255) << (8 * b);
                ts[d] += dg[d] * (1 << sh);
            }
        }
    }
#pragma unroll
    for (int d = 0; d < 4; d++)
#pragma unroll
        for (uint32_t o = 1; o < 8; o *= 2) ts[d] += __shfl_xor_sync(0xffffffffu, ts[d], o);
    if (live && u < 2) tsum[u] = u ? ts[2] * 256 + ts[3] : ts[0] * 256 + ts[1];
    if (!live) return;
#pragma unroll
    for (uint32_t d = 0; d < 4; d++) reinterpret_cast<uint4*>(rec)[h * 32 + (col * 4 + d) * 4 + t] = make_uint4(out[d][0], out[d][1], out[d][2], out[d][3]);
}

// Digit table of vector blockIdx.y; columns of vectors past the batch stay as they are (a column only reaches its own results).
template <int FMT>
__global__ void __launch_bounds__(256) block_table_kernel(const float* x, uint32_t cols, uint32_t nb, uint32_t nt, uint8_t* digits, int* tsum, float* kappa_out) {
    using F = BlkFmt<FMT>;
    __shared__ float red[8];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t v = blockIdx.y, tid = threadIdx.x;
    const float* xv = x + (size_t)v * cols;
    bool finite;
    FixedScale to_fixed;
    float kappa;
    const float amax = vec_amax<256>(xv, cols, true, red, finite);
    fixed_scale<BLK_FIX_BITS>(amax, finite, to_fixed, kappa);
    if (blockIdx.x == 0 && tid == 0) kappa_out[v] = kappa;
    const uint32_t i = blockIdx.x * 256 + tid, blk = i / 8;
    const size_t at = (size_t)blk * nt + (v >> 1);
    block_record<FMT>(xv + (size_t)blk * F::EL, blk < nb, i % 8, v & 1u, to_fixed, digits + at * F::DIG, tsum + at * 4 + (v & 1u) * 2);
}

__device__ __forceinline__ uint32_t w4(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
// Plain loads and products that are no volatile assembly: the compiler may bring operands in ahead of earlier products.
template <class V> __device__ __forceinline__ V ld(const uint8_t* p) { return *reinterpret_cast<const V*>(p); }
__device__ __forceinline__ uint32_t ld_u2(const uint8_t* p) {      // a 32-bit word at a 2-byte boundary
    const uint32_t a = smem_u32(p) & 2u;
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p - a);
    return __funnelshift_r(q[0], q[1], a * 8u);
}
__device__ __forceinline__ void mma_u8s8_k16p(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(b0));
}
__device__ __forceinline__ void mma_u8s8_k32p(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma0_u8s8_k32p(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
// Two Q1_0 blocks of rows g and g + 8 for ONE vector in eight products of 32: the first block in k slots 0 .. 15 against columns 0 .. 3, the
// second in slots 16 .. 31 against columns 4 .. 7 (their records are zero in the other four), so quad lanes 0 and 1 hold the digit sums of
// the first, 2 and 3 those of the second, and each finishes one block. About 75 instructions per 576 bytes against 120 block by block.
// With rows of whole 16 bytes the second block's signs are aligned words, the first one's lie between two.
template <bool AL>
__device__ __forceinline__ void q1_pair(const uint8_t* pA, const uint8_t* pB, const uint8_t* rec, const uint8_t* tsum, bool second, uint32_t lane, float (&acc)[2]) {
    const uint32_t t = lane & 3u, which = t >> 1;
    uint32_t a0, a1, a2, a3;
    if (AL) {
        const uint32_t *qA = reinterpret_cast<const uint32_t*>(pA) + t, *qB = reinterpret_cast<const uint32_t*>(pB) + t;
        a0 = __byte_perm(qA[0], qA[1], 0x5432); a1 = __byte_perm(qB[0], qB[1], 0x5432);
        a2 = qA[5]; a3 = qB[5];
    } else {
        a0 = ld_u2(pA + 2 + 4 * t); a1 = ld_u2(pB + 2 + 4 * t);
        a2 = ld_u2(pA + 20 + 4 * t); a3 = ld_u2(pB + 20 + 4 * t);
    }
    float dA = f16_bits_to_f32(ld<uint16_t>(pA + 18 * which)), dB = f16_bits_to_f32(ld<uint16_t>(pB + 18 * which));
    if (!second) {       // an odd number of blocks: what lies there is no block
        a2 = a3 = 0u;
        if (which) dA = dB = 0.0f;
    }
    int c0[4], c1[4];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint4 x = ld<uint4>(rec + h * 512 + lane * 16), z = ld<uint4>(rec + 1024 + h * 512 + lane * 16);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t m = 0x01010101u << (4 * h + j);
            int (&c)[4] = j & 1 ? c1 : c0;
            if (h == 0 && j < 2) mma0_u8s8_k32p(c, a0 & m, a1 & m, a2 & m, a3 & m, w4(x, j), w4(z, j));
            else mma_u8s8_k32p(c, a0 & m, a1 & m, a2 & m, a3 & m, w4(x, j), w4(z, j));
        }
    }
    const int T = (int)ld<uint32_t>(tsum + which * 16 + (t & 1u) * 4);
    const int vA = 2 * ((c0[0] + c1[0]) * 256 + (c0[1] + c1[1])) - T, vB = 2 * ((c0[2] + c1[2]) * 256 + (c0[3] + c1[3])) - T;
    acc[0] = fmaf(dA, (float)vA, acc[0]);
    acc[1] = fmaf(dB, (float)vB, acc[1]);
}

// Sums of a stage of four Q8_0 rows over V vectors: of even and odd columns in the two halves of a register, or, where eight vectors leave
// no room for twice as many registers, plain.
template <int V> struct Q8Part {
    static constexpr bool PAIRS = V <= 4;
    uint64_t two[PAIRS ? V : 1][4];
    float one[PAIRS ? 1 : V][4];
};
// One Q8_0 block of four rows (columns 4 c .. 4 c + 3 of it; p: where the rows' block begins) times V vectors `pitch` bytes apart. PHASE: p
// modulo 4, 1 if it is not known ahead.
template <int V, int PHASE>
__device__ __forceinline__ void q8_block(const uint8_t* const (&p)[4], const uint8_t* x, uint32_t pitch, uint32_t c, Q8Part<V>& part) {
    uint64_t w[4][2];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float d = f16_bits_to_f32(ld<uint16_t>(p[i]));
        uint32_t q;
        if (PHASE == 0) q = __byte_perm(ld<uint32_t>(p[i] + 4 * c), ld<uint32_t>(p[i] + 4 * c + 4), 0x5432);
        else if (PHASE == 2) q = ld<uint32_t>(p[i] + 2 + 4 * c);
        else q = ld_u2(p[i] + 2 + 4 * c);
        q ^= 0x80808080u;      // bias to unsigned
        // 0x4B000000 | byte is the float 8388608 + byte; less 8388736 it is the int8 value
        const uint64_t off = pack2(-8388736.0f, -8388736.0f), dd = pack2(d, d);
        w[i][0] = mul2(add2(pack2(__uint_as_float(__byte_perm(q, 0x4B000000u, 0x7650)), __uint_as_float(__byte_perm(q, 0x4B000000u, 0x7651))), off), dd);
        w[i][1] = mul2(add2(pack2(__uint_as_float(__byte_perm(q, 0x4B000000u, 0x7652)), __uint_as_float(__byte_perm(q, 0x4B000000u, 0x7653))), off), dd);
    }
#pragma unroll
    for (int v = 0; v < V; v++) {
        if constexpr (Q8Part<V>::PAIRS) {
            const ulonglong2 e = ld<ulonglong2>(x + v * pitch + c * 16);
#pragma unroll
            for (int i = 0; i < 4; i++) part.two[v][i] = fma2(w[i][1], e.y, fma2(w[i][0], e.x, part.two[v][i]));
        } else {
            const float4 e = ld<float4>(x + v * pitch + c * 16);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 a = unpack2(w[i][0]), b = unpack2(w[i][1]);
                part.one[v][i] = fmaf(b.y, e.w, fmaf(b.x, e.z, fmaf(a.y, e.y, fmaf(a.x, e.x, part.one[v][i]))));
            }
        }
    }
}

// AL: rows are multiples of 16 bytes, so a stage starts on a 16-byte boundary. ONE: one vector, Q1_0 blocks in pairs.
template <int FMT, int NT, bool SW, bool AL, bool ONE>
__global__ void __launch_bounds__(BLK_WARPS * 32, 1) block_rows_kernel(const __grid_constant__ BlkArgs a, const uint32_t S) {
    extern __shared__ __align__(128) uint8_t smem[];
    using F = BlkFmt<FMT>;
    __shared__ float s_red[BLK_WARPS], s_kappa[2];
    constexpr int MATS = SW ? 2 : 1, V = ONE ? 1 : 2 * NT;
    constexpr uint32_t CH = F::BB * BLK_ITEM / 16 + (AL ? 0 : 1), STAGE = 16 * F::PITCH;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3u;
    const uint32_t rank = S > 1 ? blockIdx.x % S : 0u, cl = blockIdx.x / S, ncl = gridDim.x / S;
    const uint32_t tiles = a.tile0[a.nw];
    const uint32_t t_lo = (uint32_t)((uint64_t)tiles * cl / ncl), nt_loc = (uint32_t)((uint64_t)tiles * (cl + 1) / ncl) - t_lo;
    const uint32_t all = (a.nb + BLK_ITEM - 1) / BLK_ITEM, s_lo = all * rank / S, ns = all * (rank + 1) / S - s_lo;
    const uint32_t b_lo = s_lo * BLK_ITEM, b_hi = min(a.nb, (s_lo + ns) * BLK_ITEM), nblk = b_hi - b_lo;
    const uint32_t bar = smem_u32(smem), ring = bar + BLK_HDR + warp * a.stages * STAGE;
    const uint8_t* const tab = smem + BLK_HDR + BLK_WARPS * a.stages * STAGE;
    const uint8_t* const tsm = smem + a.tsum_off;
    float* mainp = reinterpret_cast<float*>(smem + a.main_off);     // [mat][tile][16 rows][2 NT]
    float* head = reinterpret_cast<float*>(smem + a.head_off);      // [warp][16 rows][2 NT]
    if (tid == 0) { mbar_init(bar, 1); mbar_fence_init(); }
    __syncthreads();
    pdl_launch_dependents();

    const uint32_t items = MATS * nt_loc * ns;
    const uint32_t i_lo = items * warp / BLK_WARPS, i_hi = items * (warp + 1) / BLK_WARPS;
    auto matrix_of = [&](uint32_t tile, uint32_t& s, const uint8_t*& w, uint32_t& r0) {     // tile: gate tiles, then up tiles
        const bool up = SW && tile >= nt_loc;
        const uint32_t tl = t_lo + (up ? tile - nt_loc : tile);
        s = 0;
        if (!SW) while (s + 1 < a.nw && tl >= a.tile0[s + 1]) s++;
        w = up ? a.up : a.w[s];
        r0 = (tl - a.tile0[s]) * 16;
    };
    // Where this lane's 16-byte pieces of a stage lie relative to the tile and the slot: a stage is a whole number of them and so are 16
    // rows, so this is the same for all tiles but a matrix's last one, and a piece costs a few additions and the copy.
    static_assert(F::BB * BLK_ITEM % 16 == 0, "stages keep the alignment of the rows");
    constexpr uint32_t PIECES = (16 * CH + 31) / 32;
    uint32_t rel[PIECES];
#pragma unroll
    for (uint32_t j = 0; j < PIECES; j++) {
        const uint32_t i = j * 32 + lane, r = i / CH, c = i - r * CH;
        rel[j] = ((r * a.row_bytes) & ~15u) + c * 16;
    }
    const uint32_t inside = 16 + (CH * 16 + a.row_bytes - 1) / a.row_bytes;      // rows from a tile's first one on that its whole stages may touch
    uint32_t l_item = i_lo, l_tile = i_lo / ns, l_seg = i_lo - l_tile * ns, l_slot = 0;
    const uint8_t *lw = nullptr, *lp = nullptr;      // matrix; this stage's columns of the tile's first row
    uint32_t ls = 0, lr0 = 0;
    auto to_tile = [&]() {
        matrix_of(l_tile, ls, lw, lr0);
        lp = lw + (uint64_t)lr0 * a.row_bytes + (uint64_t)(s_lo + l_seg) * (BLK_ITEM * F::BB);
    };
    if (i_lo < i_hi) to_tile();
    auto fetch = [&]() {
        if (l_item < i_hi) {
            const uint32_t dst = ring + l_slot * STAGE;
            if (lr0 + inside <= a.rows[ls]) {
#pragma unroll
                for (uint32_t j = 0; j < PIECES; j++) {
                    if (16 * CH % 32 && j * 32 + lane >= 16 * CH) continue;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (j * 32 + lane) * 16 + (j * 32 + lane) / CH * (F::PITCH - CH * 16)), "l"(lp + rel[j]) : "memory");
                }
            } else {        // rows past the last repeat it, nothing past the matrix is read
                const uint64_t total = (uint64_t)a.rows[ls] * a.row_bytes;
                const uint32_t at = (s_lo + l_seg) * (BLK_ITEM * F::BB);
#pragma unroll 1
                for (uint32_t i = lane; i < 16 * CH; i += 32) {
                    const uint32_t r = i / CH, c = i - r * CH;
                    const uint64_t off = (((uint64_t)min(lr0 + r, a.rows[ls] - 1) * a.row_bytes + at) & ~(uint64_t)15) + c * 16;
                    const uint32_t n = off < total ? (uint32_t)min((uint64_t)16, total - off) : 0u;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + r * F::PITCH + c * 16), "l"(n ? lw + off : lw), "r"(n) : "memory");
                }
            }
            l_item++;
            lp += BLK_ITEM * F::BB;
            if (++l_seg == ns) { l_seg = 0; l_tile++; if (l_item < i_hi) to_tile(); }
            if (++l_slot == a.stages) l_slot = 0;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (uint32_t k = 0; k + 1 < a.stages; k++) fetch();

    pdl_wait();
    bool ok = true;
    if constexpr (FMT != 0 && NT == 1) {
        // one or two vectors: every CTA makes the digits of its columns itself, which saves the launch of the table kernel in between
        uint8_t* const dtab = smem + BLK_HDR + BLK_WARPS * a.stages * STAGE;
        int* const dsum = reinterpret_cast<int*>(smem + a.tsum_off);
        for (uint32_t v = 0; v < a.batch; v++) {
            const float* xv = a.x + (size_t)v * a.nb * F::EL;
            bool finite;
            FixedScale to_fixed;
            float kappa;
            const float amax = vec_amax<BLK_WARPS * 32>(xv, a.nb * F::EL, true, s_red, finite);
            fixed_scale<BLK_FIX_BITS>(amax, finite, to_fixed, kappa);
            if (tid == 0) s_kappa[v] = kappa;
            for (uint32_t i = tid; i < ((nblk * 8 + 31) & ~31u); i += BLK_WARPS * 32) {
                if (ONE) {       // odd blocks in columns 4 .. 7, zeros in the others
                    const uint32_t b = i / 8, col = b & 1u;
                    uint8_t* rec = dtab + b * F::DIG;
                    if (b < nblk)
#pragma unroll
                        for (uint32_t d = 0; d < 4; d++) reinterpret_cast<uint4*>(rec)[((i >> 2) & 1u) * 32 + ((1 - col) * 4 + d) * 4 + (i & 3u)] = make_uint4(0u, 0u, 0u, 0u);
                    block_record<FMT>(xv + (size_t)(b_lo + b) * F::EL, b < nblk, i % 8, col, to_fixed, rec, dsum + b * 4);
                    continue;
                }
                block_record<FMT>(xv + (size_t)(b_lo + i / 8) * F::EL, i / 8 < nblk, i % 8, v, to_fixed, dtab + (i / 8) * F::DIG, dsum + (i / 8) * 4 + v * 2);
            }
        }
        __syncthreads();
    } else {
        if (tid == 0) {
            if (FMT == 0) {      // the vectors themselves; those past the batch stay as they are
                mbar_arrive_expect_tx(bar, a.batch * nblk * 128u);
                for (uint32_t v = 0; v < a.batch; v++) bulk_g2s(smem_u32(tab) + v * nblk * 128u, a.x + ((size_t)v * a.nb + b_lo) * 32, nblk * 128u, bar);
            } else {
                const uint32_t db = nblk * NT * F::DIG, tb = nblk * NT * 16u;
                mbar_arrive_expect_tx(bar, db + tb);
                bulk_g2s(smem_u32(tab), a.digits + (size_t)b_lo * NT * F::DIG, db, bar);
                bulk_g2s(smem_u32(tsm), a.tsum + (size_t)b_lo * NT * 4, tb, bar);
            }
        }
        ok = mbar_wait_limit(bar, 0, a.wait_limit > 0 ? a.wait_limit : WAIT_CYCLE_LIMIT);
        if (!ok && lane == 0) atomicCAS(a.status, 0, KERR_WAIT_FULL);
    }

    float acc[NT][2] = {}, accf[FMT == 0 ? V : 1][4] = {};     // Q8_0: rows lane / 8 + 4 i, all vectors
    uint32_t tile = i_lo / ns, seg = i_lo - tile * ns, slot = 0, padA = 0, padB = 0, pad[4] = {0u, 0u, 0u, 0u};
    bool mid = seg != 0;                     // this warp took the tile up in its middle
    auto pads = [&]() {
        if (AL) return;
        uint32_t s, r0;
        const uint8_t* w;
        matrix_of(tile, s, w, r0);
        if (FMT == 0) {
#pragma unroll
            for (int i = 0; i < 4; i++) pad[i] = (min(r0 + (lane >> 3) + 4 * i, a.rows[s] - 1) * a.row_bytes) & 15u;
            return;
        }
        padA = (min(r0 + g, a.rows[s] - 1) * a.row_bytes) & 15u;
        padB = (min(r0 + g + 8, a.rows[s] - 1) * a.row_bytes) & 15u;
    };
    if (i_lo < i_hi) pads();
    auto flush = [&]() {
        float* dst = mid ? head + warp * (16 * 2 * NT) : mainp + (size_t)((tile >= nt_loc ? a.tiles_max + (tile - nt_loc) : tile) * 16) * (2 * NT);
        if constexpr (FMT == 0) {
#pragma unroll
            for (int v = 0; v < V; v++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    float y = accf[v][i];
#pragma unroll
                    for (int o = 1; o < 8; o *= 2) y += __shfl_xor_sync(0xffffffffu, y, o);
                    if ((lane & 7u) == (uint32_t)v) dst[((lane >> 3) + 4 * i) * (2 * NT) + v] = y;
                    accf[v][i] = 0.0f;
                }
            mid = false;
            return;
        }
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float f = (t & 1u) ? acc[n][h] : acc[n][h] * 65536.0f;
                float y = f + __shfl_xor_sync(0xffffffffu, f, 1);
                if (ONE) y += __shfl_xor_sync(0xffffffffu, y, 2);
                if (ONE ? t == 0 : !(t & 1u)) dst[(g + 8 * h) * (2 * NT) + 2 * n + (t >> 1)] = y;
                acc[n][h] = 0.0f;
            }
        mid = false;
    };
    for (uint32_t it = i_lo; ok && it < i_hi; it++) {
        if (a.stages == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
        else if (a.stages == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 2;" ::: "memory");
        __syncwarp();                        // the stage is in for every lane, and every lane is done with the one before
        fetch();
        const uint8_t* const stage = smem + BLK_HDR + (warp * a.stages + slot) * STAGE;
        const uint8_t *const rowA = stage + g * F::PITCH + padA, *const rowB = stage + (g + 8) * F::PITCH + padB;
        if (++slot == a.stages) slot = 0;
        const uint32_t b0 = seg * BLK_ITEM, nbi = min(BLK_ITEM, nblk - b0);
        if constexpr (FMT == 0) {
            const uint8_t* p[4];
#pragma unroll
            for (int i = 0; i < 4; i++) p[i] = stage + ((lane >> 3) + 4 * i) * F::PITCH + pad[i];
            const uint8_t* x = tab + b0 * 128u;
            Q8Part<V> part = {};               // a stage's sum: shorter chains of f32 additions than a row of them
            auto next = [&](uint32_t n) {
#pragma unroll
                for (int i = 0; i < 4; i++) p[i] += n * F::BB;
                x += n * 128;
            };
            if (AL) {                          // whole stages of blocks that begin at 0, 2, 0, 2 .. modulo 4
#pragma unroll 1
                for (uint32_t b = 0; b < BLK_ITEM; b += 2) {
                    q8_block<V, 0>(p, x, nblk * 128u, lane & 7u, part);
                    next(1);
                    q8_block<V, 2>(p, x, nblk * 128u, lane & 7u, part);
                    next(1);
                }
            } else {
#pragma unroll 1
                for (uint32_t b = 0; b < nbi; b++) { q8_block<V, 1>(p, x, nblk * 128u, lane & 7u, part); next(1); }
            }
#pragma unroll
            for (int v = 0; v < V; v++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if constexpr (Q8Part<V>::PAIRS) { const float2 y = unpack2(part.two[v][i]); accf[v][i] += y.x + y.y; }
                    else accf[v][i] += part.one[v][i];
                }
            if (++seg == ns) { flush(); seg = 0; tile++; if (it + 1 < i_hi) pads(); }
            continue;
        }
        const uint8_t *const rec = tab + b0 * (NT * F::DIG), *const trec = tsm + b0 * (NT * 16u) + t * 4;
        auto block = [&](uint32_t b) {
            if constexpr (FMT != 0) {
                const uint8_t *const pA = rowA + b * F::BB, *const pB = rowB + b * F::BB;
                const float dA = f16_bits_to_f32(ld<uint16_t>(pA)), dB = f16_bits_to_f32(ld<uint16_t>(pB));
                int c[NT][2][4] = {};        // even and odd bits: two chains
                if constexpr (FMT == 1) {
                    const uint32_t a0 = ld_u2(pA + 2 + 4 * t), a1 = ld_u2(pB + 2 + 4 * t);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        uint4 x[NT];
#pragma unroll
                        for (int n = 0; n < NT; n++) x[n] = ld<uint4>(rec + (b * NT + n) * F::DIG + h * 512 + lane * 16);
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const uint32_t m = 0x01010101u << (4 * h + j), m0 = a0 & m, m1 = a1 & m;
#pragma unroll
                            for (int n = 0; n < NT; n++) mma_u8s8_k16p(c[n][j & 1], m0, m1, w4(x[n], j));
                        }
                    }
                } else {
                    const uint32_t a0 = ld_u2(pA + 2 + 4 * t), a1 = ld_u2(pB + 2 + 4 * t), a2 = ld_u2(pA + 18 + 4 * t), a3 = ld_u2(pB + 18 + 4 * t);
                    uint4 x[NT], z[NT];
#pragma unroll
                    for (int n = 0; n < NT; n++) {
                        x[n] = ld<uint4>(rec + (b * NT + n) * F::DIG + lane * 16);
                        z[n] = ld<uint4>(rec + (b * NT + n) * F::DIG + 512 + lane * 16);
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const uint32_t m = 0x03030303u << (2 * j), m0 = a0 & m, m1 = a1 & m, m2 = a2 & m, m3 = a3 & m;
#pragma unroll
                        for (int n = 0; n < NT; n++) mma_u8s8_k32p(c[n][j & 1], m0, m1, m2, m3, w4(x[n], j), w4(z[n], j));
                    }
                }
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    const int T = (int)ld<uint32_t>(trec + (b * NT + n) * 16);
                    int vA = (c[n][0][0] + c[n][1][0]) * 256 + (c[n][0][1] + c[n][1][1]), vB = (c[n][0][2] + c[n][1][2]) * 256 + (c[n][0][3] + c[n][1][3]);
                    vA = (FMT == 1 ? 2 * vA : vA) - T;
                    vB = (FMT == 1 ? 2 * vB : vB) - T;
                    acc[n][0] = fmaf(dA, (float)vA, acc[n][0]);
                    acc[n][1] = fmaf(dB, (float)vB, acc[n][1]);
                }
            }
        };
        if constexpr (ONE && FMT == 1) {
            if (nbi == BLK_ITEM) {
#pragma unroll
                for (uint32_t b = 0; b < BLK_ITEM; b += 2) q1_pair<AL>(rowA + b * F::BB, rowB + b * F::BB, rec + b * F::DIG, trec + b * 16 - t * 4, true, lane, acc[0]);
            } else
#pragma unroll 1
            for (uint32_t b = 0; b < nbi; b += 2) q1_pair<AL>(rowA + b * F::BB, rowB + b * F::BB, rec + b * F::DIG, trec + b * 16 - t * 4, b + 1 < nbi, lane, acc[0]);
        } else if (nbi == BLK_ITEM) {
#pragma unroll 2
            for (uint32_t b = 0; b < BLK_ITEM; b++) block(b);
        } else {
#pragma unroll 1
            for (uint32_t b = 0; b < nbi; b++) block(b);
        }
        if (++seg == ns) { flush(); seg = 0; tile++; if (it + 1 < i_hi) pads(); }
    }
    if (ok && seg != 0 && i_lo < i_hi) flush();
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // parts of tiles that another warp began, in the order of the warps
    if (tid < 16 * 2 * NT) {
        for (uint32_t w = 1; w < (uint32_t)BLK_WARPS; w++) {
            const uint32_t lo = items * w / BLK_WARPS, hi = items * (w + 1) / BLK_WARPS, tl = lo / ns;
            if (lo < hi && lo != tl * ns) mainp[(size_t)((tl >= nt_loc ? a.tiles_max + (tl - nt_loc) : tl) * 16) * (2 * NT) + tid] += head[w * (16 * 2 * NT) + tid];
        }
    }
    if (S > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
    const uint32_t R = nt_loc * 16, outs = R * a.batch;
    const uint32_t main_s = bar + a.main_off;
    unsigned long long key = 0ull;
    for (uint32_t i = rank * (BLK_WARPS * 32) + tid; ok && i < outs; i += S * (BLK_WARPS * 32)) {
        const uint32_t v = i / R, lr = i - v * R, tl = t_lo + lr / 16;
        uint32_t s = 0;
        if (!SW) while (s + 1 < a.nw && tl >= a.tile0[s + 1]) s++;
        const uint32_t row = (tl - a.tile0[s]) * 16 + lr % 16;
        if (row >= a.rows[s]) continue;
        float f[MATS];
#pragma unroll
        for (int q = 0; q < MATS; q++) {
            const uint32_t at = main_s + ((q * a.tiles_max * 16 + lr) * (2 * NT) + v) * 4;
            float y = ldsf(at);
            if (S > 1) {
                for (uint32_t r = 0; r < S; r++) {
                    uint32_t remote;
                    float p;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(r));
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(p) : "r"(remote) : "memory");
                    y = r ? y + p : p;
                }
            }
            f[q] = FMT == 0 ? y : (NT == 1 ? s_kappa[v] : __ldg(a.kappa + v)) * y;
        }
        float r = SW ? silu_ref(f[0]) * f[MATS - 1] : f[0];
        const uint32_t yi = a.y_off[s] + row;
        const size_t at = (size_t)v * a.y_stride + yi;
        if (a.resid != nullptr) r = __fadd_rn(__ldcg(a.resid + at), r);
        a.y[at] = r;
        const uint32_t b = __float_as_uint(r), ordered = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
        const unsigned long long k = r == r ? ((unsigned long long)ordered << 32) | (0xFFFFFFFFu - yi) : 0ull;
        key = k > key ? k : key;
    }
    if (a.argmax_key != nullptr) stream_argmax(a.argmax_key, key, lane);
    if (S > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

template <int FMT, int NT, bool SW, bool AL, bool ONE>
int plan_and_launch_one(BlkArgs a, const LaunchCfg& cfg, bool dry) {
    using F = BlkFmt<FMT>;
    static bool attr_done[64] = {};
    static int clusters[64][4] = {};
    auto kern = block_rows_kernel<FMT, NT, SW, AL, ONE>;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return ALICE_E_CUDA;
    if (!attr_done[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BLK_SMEM) != cudaSuccess) return ALICE_E_CUDA;
        attr_done[dev] = true;
    }
    const uint32_t sms = (uint32_t)std::max(cfg.num_sms, 1), tiles = a.tile0[a.nw], all = (a.nb + BLK_ITEM - 1) / BLK_ITEM;
    cudaLaunchConfig_t lc = {};
    lc.blockDim = dim3(BLK_WARPS * 32); lc.stream = cfg.stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    for (uint32_t S = 1, l2 = 0; S <= 8 && S <= all; S *= 2, l2++) {
        uint32_t ncl = sms;
        if (S > 1) {      // a cluster's CTAs sit in one GPC: what the chip holds at once is asked for, once per kernel and device
            int& known = clusters[dev][l2];
            if (!known) {
                at[0].val.clusterDim.x = S;
                lc.attrs = at; lc.numAttrs = 1; lc.gridDim = dim3(sms / S * S); lc.dynamicSmemBytes = BLK_SMEM;
                int n = 0;
                if (sms < S || cudaOccupancyMaxActiveClusters(&n, kern, &lc) != cudaSuccess || n < 1) { cudaGetLastError(); break; }
                known = n;
            }
            ncl = std::min<uint32_t>((uint32_t)known, sms / S);
        }
        ncl = std::min(ncl, tiles);
        const uint32_t per = (tiles + ncl - 1) / ncl, slice = (all + S - 1) / S * BLK_ITEM;
        const size_t dig = (size_t)slice * NT * F::DIG, ts = F::T ? (size_t)slice * NT * 16 : 0, mn = (size_t)(SW ? 2 : 1) * per * 16 * 2 * NT * 4,
                     hd = (size_t)BLK_WARPS * 16 * 2 * NT * 4, stage = (size_t)BLK_WARPS * 16 * F::PITCH, fixed = BLK_HDR + dig + ts + mn + hd;
        if (fixed + 2 * stage > BLK_SMEM) continue;
        // fewer tiles than half the SMs: let more CTAs share a tile's columns
        if (S < 8 && tiles * S * 2 <= sms && all >= 2 * S) continue;
        if (dry) return ALICE_OK;
        a.stages = (uint32_t)std::min<size_t>(4, (BLK_SMEM - fixed) / stage);
        a.tiles_max = per;
        a.tsum_off = (uint32_t)(BLK_HDR + a.stages * stage + dig);
        a.main_off = (uint32_t)(a.tsum_off + ts); a.head_off = (uint32_t)(a.main_off + mn);
        at[0].val.clusterDim.x = S;
        lc.gridDim = dim3(ncl * S); lc.dynamicSmemBytes = fixed + a.stages * stage;
        lc.attrs = S > 1 ? at : at + 1;
        lc.numAttrs = (S > 1 ? 1 : 0) + (cfg.pdl ? 1 : 0);
        return cudaLaunchKernelEx(&lc, kern, a, S) == cudaSuccess ? ALICE_OK : ALICE_E_CUDA;
    }
    return ALICE_E_SHAPE;
}

template <int FMT, int NT, bool SW, bool AL>
int plan_and_launch(const BlkArgs& a, const LaunchCfg& cfg, bool dry) {
    if constexpr (FMT != 2 && NT == 1)
        if (a.batch == 1) return plan_and_launch_one<FMT, NT, SW, AL, true>(a, cfg, dry);
    return plan_and_launch_one<FMT, NT, SW, AL, false>(a, cfg, dry);
}

template <int FMT, int NT>
int launch_nt(const BlkArgs& a, const LaunchCfg& cfg, bool dry) {
    const bool al = a.row_bytes % 16 == 0;
    if (a.up) return al ? plan_and_launch<FMT, NT, true, true>(a, cfg, dry) : plan_and_launch<FMT, NT, true, false>(a, cfg, dry);
    return al ? plan_and_launch<FMT, NT, false, true>(a, cfg, dry) : plan_and_launch<FMT, NT, false, false>(a, cfg, dry);
}
uint32_t pairs_of(uint32_t batch) { return batch <= 2 ? 1u : batch <= 4 ? 2u : 4u; }

template <int FMT>
int launch_blk(BlkArgs a, const GemvOp& op, const LaunchCfg& cfg, bool dry) {
    using F = BlkFmt<FMT>;
    const uint32_t nt = pairs_of(op.batch), cols = op.w[0]->cols;
    a.nb = cols / F::EL;
    const size_t dig = (size_t)a.nb * nt * F::DIG, ts = F::T ? (size_t)a.nb * nt * 16 : 0;
    a.x = op.x;
    const bool table = F::T && nt > 1;
    if (!dry && table) {
        if (!op.prep || ((uintptr_t)op.prep & 15) || dig + ts + 64 > op.prep_bytes) return ALICE_E_SHAPE;
        uint8_t* base = static_cast<uint8_t*>(op.prep);
        a.digits = base; a.tsum = reinterpret_cast<const int*>(base + dig); a.kappa = reinterpret_cast<const float*>(base + dig + ts);
    }
    auto rows = [&](bool plan) { return nt == 1 ? launch_nt<FMT, 1>(a, cfg, plan) : nt == 2 ? launch_nt<FMT, 2>(a, cfg, plan) : launch_nt<FMT, 4>(a, cfg, plan); };
    const int rc = rows(true);
    if (rc || dry) return rc;
    if (!table) return rows(false);
    cudaLaunchConfig_t lc = {};
    const uint32_t per_vec = a.nb * 8u;
    lc.gridDim = dim3((per_vec + 255) / 256, op.batch); lc.blockDim = dim3(256); lc.stream = cfg.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at; lc.numAttrs = cfg.pdl ? 1 : 0;
    if (cudaLaunchKernelEx(&lc, block_table_kernel<F::T ? FMT : 1>, op.x, cols, a.nb, nt, const_cast<uint8_t*>(a.digits), const_cast<int*>(a.tsum), const_cast<float*>(a.kappa)) != cudaSuccess)
        return ALICE_E_CUDA;
    return rows(false);
}

}  // namespace

size_t blocks_prep_bytes(uint32_t cols, uint32_t batch) {
    return (size_t)((cols + 127) / 128) * pairs_of(batch) * (1024 + 16) + 256;
}

int launch_blocks(const GemvOp& op, const LaunchCfg& cfg, bool dry, uint32_t* launches) {
    if (launches) *launches = 1;
    const WeightDesc& w0 = *op.w[0];
    if ((w0.fmt != WF_Q8_0 && w0.fmt != WF_Q1_0 && w0.fmt != WF_Q2_0) || op.npeers || op.norm_w || op.batch == 0 || op.batch > 8 || (op.argmax_key && op.batch > 1)) return ALICE_E_SHAPE;
    if (op.nw < 1 || op.nw > 3 || (op.up && op.nw != 1) || !op.y || !op.x || ((uintptr_t)op.x & 15)) return ALICE_E_SHAPE;
    BlkArgs a = {};
    uint32_t total = 0;
    for (uint32_t i = 0; i < op.nw; i++) {
        const WeightDesc* w = op.w[i];
        if (!w || !w->data || !w->rows || ((uintptr_t)w->data & 15) || w->fmt != w0.fmt || w->cols != w0.cols || w->row_bytes != w0.row_bytes) return ALICE_E_SHAPE;
        a.w[i] = w->data; a.rows[i] = w->rows; a.y_off[i] = op.y_off[i];
        a.tile0[i + 1] = a.tile0[i] + (w->rows + 15) / 16;
        total += w->rows;
    }
    if (op.up) {
        const WeightDesc& u = *op.up;
        if (u.fmt != w0.fmt || u.rows != w0.rows || u.cols != w0.cols || u.row_bytes != w0.row_bytes || !u.data || ((uintptr_t)u.data & 15)) return ALICE_E_SHAPE;
        a.up = u.data;
    }
    a.nw = op.nw; a.row_bytes = w0.row_bytes;
    a.y = op.y; a.resid = op.resid; a.y_stride = op.y_stride ? op.y_stride : total; a.batch = op.batch;
    a.argmax_key = op.argmax_key; a.status = cfg.status; a.wait_limit = op.wait_limit;
    return w0.fmt == WF_Q8_0 ? launch_blk<0>(a, op, cfg, dry) : w0.fmt == WF_Q1_0 ? launch_blk<1>(a, op, cfg, dry) : launch_blk<2>(a, op, cfg, dry);
}

}  // namespace alice

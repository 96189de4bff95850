// Ternary planes and packed codes times three to eight vectors on the fifth-generation tensor cores.
//
// The int8 mma.sync of csrc/gemv_planes.cu takes 8 clk for 16 rows x 32 columns and eight digit columns, and every warp reads all B fragments from shared
// memory: eight vectors (32 digit columns) cost twice one. tcgen05 kind::i8 takes 16 clk for 128 x 32 x 32, its A operand from tensor memory, where the
// warps that unpack put a row a lane, B from shared memory, where a chunk of 16 k of all digits lies without padding.
//
// One CTA an SM, 21 warps: 4 copy (cp.async, 64-byte segments of 128 rows), 16 unpack, 1 multiplies (an elected lane: a lane picked by its number takes 44
// clk to issue a product). The unpacking warps are four groups, each at every fourth half of a segment, so that some are unpacking while others
// wait. A cluster shares the columns, so that the digits of a CTA's fit beside its ring; accumulators of all of a CTA's tiles stay in tensor memory until the
// end, where a sum's digits meet in 64 bits and the CTAs of a cluster add theirs. Rows are dealt evenly, not in whole tiles.
//
// Measured against csrc/gemv_planes.cu, eight vectors, digit tables included: 28672 x 8192 37.5 -> 24.5 us, 8192 x 28672 45.3 -> 29.8, 8192 x 8192 19.1 -> 12.3; gate
// and up of 28672 x 8192 64.1 -> 52.9. What bounds it: the hand-overs between the warps and the start and end of a launch (7 us). No unit is near its
// peak: ALU 49 % (14 bit operations for 32 weights, one every other clk and SM quarter), tensor pipe 17, HBM 24, shared memory 14.
#include <algorithm>

#include "../../include/alice_cuda.h"
#include "digits_dev.cuh"
#include "gemv_mma.cuh"
#include "gemv_planes.cuh"
#include "planes_dev.cuh"
#include "tc_dev.cuh"

namespace alice {
namespace {

// Warps: 16 unpack (four groups of 128 rows x a piece of 16 bytes each), 4 copy, 1 multiplies.
constexpr uint32_t PT_UNPACK = 512, PT_COPY = 128, PT_THREADS = PT_UNPACK + PT_COPY + 32;
constexpr uint32_t PT_TILES = 32, PT_STAGES = 8, PT_SLOTS = 4, PT_D = 256;       // accumulators: columns 256 and up of tensor memory
constexpr uint32_t PT_SMEM = 225 * 1024, PT_SMEM_MIN = 120 * 1024;              // never two CTAs on an SM: each takes all of its tensor memory
constexpr int KERR_PT_WAIT = 7;

struct PtArgs {
    const uint8_t* w[3];
    const float* scale[3];
    uint32_t rows[3], y_off[3], row0[4], nw;
    const uint8_t* up;
    const float* up_scale;
    uint32_t row_bytes, plane, segs;             // bytes of a row and of a plane; 64-byte segments of a plane
    const uint4* table;                          // [16 k][vector][digit][16 bytes]
    const float* kappa;
    float* y;
    const float* resid;
    uint32_t y_stride, batch;
    uint32_t row_lo, nrows, stages, tab_off;     // rows of this launch; shared memory: ring | table
    int* status;
    long long wait_limit;
};

struct PtTile { const uint8_t* base; uint32_t n, at; };      // up to 128 rows of a matrix, the first is row `at` of the CTA's

template <int PL> struct PtGeom {      // PL: planes of a row (2: pos | neg, 1: codes)
    static constexpr uint32_t PITCH = PL == 2 ? 144 : 80, STAGE = 128 * PITCH;    // an odd number of 16-byte pieces
    static constexpr uint32_t CP = PL == 2 ? 8 : 4, AW = 4 * CP;                  // B chunks of 16 k and words of A of a 16-byte piece
};

// A weight w (-1, 0 or 1) enters as 1 + w in a two-bit field, worth 4^k at place k of its byte: the fields of 32 weights (a word of either plane) take
// six bit operations, and one mask cuts the operand of four weights out of them (a signed byte of its own takes two masks and a multiplication).
// What the ones add up to, over all columns, is taken off a row's sum in integers.
struct PlaneFields { uint32_t x, y; };      // of 1 + w: one of its two bits is set, both are
__device__ __forceinline__ PlaneFields plane_fields(uint32_t p, uint32_t n) { return {p ^ ~n, p & ~n}; }
__device__ __forceinline__ uint32_t even_fields(const PlaneFields& f) { return (f.x & 0x55555555u) | (f.y << 1 & 0xaaaaaaaau); }
__device__ __forceinline__ uint32_t odd_fields(const PlaneFields& f) { return (f.x >> 1 & 0x55555555u) | (f.y & 0xaaaaaaaau); }
// The same of 16 codes 00 = 0, 01 = +1, 11 = -1.
__device__ __forceinline__ uint32_t code_fields(uint32_t w) { return ~w & (w << 1 | 0x55555555u); }
__device__ __forceinline__ uint32_t field_bytes(uint32_t f, int k) { return f & (0x03030303u << (2 * k)); }
// What the ones of one chunk of 16 digit bytes (places 0 .. 3) add up to, and the worth of digit d in fixed-point units.
__device__ __forceinline__ int field_total(const uint4& c) {
    return dp4a_ss(c.x, 0x01010101u, 0) + 4 * dp4a_ss(c.y, 0x01010101u, 0) + 16 * dp4a_ss(c.z, 0x01010101u, 0) + 64 * dp4a_ss(c.w, 0x01010101u, 0);
}
__device__ __forceinline__ long long digit_worth(uint32_t d) { return 1ll << (7 * (3 - d)); }

// Digits of one chunk (16 k) of one vector: word w of a 16-byte piece of weights; planes: places 0 .. 3 of the even (h = 0) or odd columns of its four
// bytes, codes: the four places of its four bytes. Activations are rounded as csrc/gemv_planes.cu rounds them (to 2^j units for bit j of a byte, 2^6 for
// bit 7), so a vector's results do not depend on how many go with it; 4^k of an odd column's place is 2^j / 2, so twice the rounded number is stored.
template <int PL>
__device__ __forceinline__ void pt_digits(const float* x, uint32_t cols, bool vec4, const FixedScale sc, uint32_t chunk, uint4* to) {
    constexpr uint32_t E = PL == 2 ? 8 : 4;             // columns of a byte
    const uint32_t piece = chunk / PtGeom<PL>::CP, c = chunk % PtGeom<PL>::CP, word = PL == 2 ? c >> 1 : c, h = PL == 2 ? c & 1u : 0u;
    uint32_t out[4][4] = {};
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) {
        const uint32_t e = (piece * 16 + word * 4 + i) * E;
        float xe[E];
#pragma unroll
        for (uint32_t k = 0; k < E; k += 4) {
            float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
            if (vec4) {
                if (e + k < cols) q = __ldcg(reinterpret_cast<const float4*>(x + e + k));
            } else {
                if (e + k < cols) q.x = __ldcg(x + e + k);
                if (e + k + 1 < cols) q.y = __ldcg(x + e + k + 1);
                if (e + k + 2 < cols) q.z = __ldcg(x + e + k + 2);
                if (e + k + 3 < cols) q.w = __ldcg(x + e + k + 3);
            }
            xe[k] = q.x; xe[k + 1] = q.y; xe[k + 2] = q.z; xe[k + 3] = q.w;
        }
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {
            const int j = 2 * k + (PL == 2 && h ? 1 : 0), sh = min(j, 6);
            const float v = PL == 2 ? (h ? xe[(2 * k + 1) % E] : xe[2 * k % E]) : xe[k % E];
            int f = (to_units(v, sc) + ((1 << sh) >> 1)) >> sh;
            if ((j & 1) && j < 7) f *= 2;
            uint8_t dg[193];          // digits land 64 apart
            mma_store_digits(dg, f);
#pragma unroll
            for (int d = 0; d < 4; d++) out[d][k] |= (uint32_t)dg[64 * d] << (8 * i);
        }
    }
#pragma unroll
    for (int d = 0; d < 4; d++) to[d] = make_uint4(out[d][0], out[d][1], out[d][2], out[d][3]);
}

template <int PL>
__global__ void __launch_bounds__(256) plane_tc_table_kernel(const float* x, uint32_t cols, uint32_t batch, uint32_t chunks, uint4* table, float* kappa_out) {
    __shared__ float red[8];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t v = blockIdx.y, tid = threadIdx.x, c = blockIdx.x * 256 + tid;
    const float* xv = x + (size_t)v * cols;
    const bool vec4 = can_vec4(xv, cols);
    bool finite;
    FixedScale sc;
    float kappa;
    const float amax = vec_amax<256>(xv, cols, vec4, red, finite);
    fixed_scale<MMA_FIX_BITS>(amax, finite, sc, kappa);
    if (blockIdx.x == 0 && tid == 0) kappa_out[v] = kappa;
    if (c < chunks) pt_digits<PL>(xv, cols, vec4, sc, c, table + ((size_t)c * batch + v) * 4);
}

__device__ __forceinline__ void mma_u8s8_ta(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool acc) {
    asm volatile("{ .reg .pred p; setp.ne.u32 p, %4, 0; tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p; }" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"((uint32_t)acc) : "memory");
}
__device__ __forceinline__ void tmem_get4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n\ttcgen05.wait::ld.sync.aligned;" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// N: columns of B, four to a vector
template <int N, int PL, bool SW>
__global__ void __launch_bounds__(PT_THREADS, 1) plane_tc_kernel(const __grid_constant__ PtArgs a, const uint32_t S) {
    extern __shared__ __align__(128) uint8_t smem[];
    using G = PtGeom<PL>;
    __shared__ __align__(8) uint64_t full_[PT_STAGES], empty_[PT_STAGES], afull_[PT_SLOTS], aempty_[PT_SLOTS], done_, tab_;
    __shared__ PtTile tiles[PT_TILES];
    __shared__ uint32_t tmem_base;
    __shared__ __align__(8) unsigned long long s_total[8];      // what the ones of the fields add to the sums of this CTA's columns, per vector
    constexpr uint32_t MATS = SW ? 2 : 1;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = S > 1 ? blockIdx.x % S : 0u, cl = blockIdx.x / S, ncl = gridDim.x / S;
    const uint32_t r_lo = a.row_lo + (uint32_t)((uint64_t)a.nrows * cl / ncl), R = a.row_lo + (uint32_t)((uint64_t)a.nrows * (cl + 1) / ncl) - r_lo;
    const uint32_t s_lo = a.segs * rank / S, ns = a.segs * (rank + 1) / S - s_lo;
    const uint32_t ring = smem_u32(smem);
    auto bar = [](uint64_t* b, uint32_t i) { return smem_u32(b + i); };
    const long long limit = a.wait_limit > 0 ? a.wait_limit : WAIT_CYCLE_LIMIT;

    // this CTA's tiles: the rows it has of every matrix in pieces of nearly equal height; with SwiGLU gate and up of a piece in turn
    uint32_t ntiles = 0;
    for (uint32_t s = 0; s < a.nw; s++) {
        const uint32_t lo = max(r_lo, a.row0[s]), hi = min(r_lo + R, a.row0[s + 1]);
        if (lo >= hi) continue;
        const uint32_t len = hi - lo, c = (len + 127) / 128;
        if (tid >= ntiles && tid < ntiles + c * MATS) {
            const uint32_t k = (tid - ntiles) / MATS, up = (tid - ntiles) % MATS, f = len * k / c, n = len * (k + 1) / c - f;
            tiles[tid] = PtTile{(up ? a.up : a.w[s]) + (uint64_t)(lo - a.row0[s] + f) * a.row_bytes, n, up * R + (lo - r_lo) + f};
        }
        ntiles += c * MATS;
    }
    if (tid == 64) {
        for (uint32_t i = 0; i < a.stages; i++) { mbar_init(bar(full_, i), PT_COPY); mbar_init(bar(empty_, i), 8); }
        for (uint32_t i = 0; i < PT_SLOTS; i++) { mbar_init(bar(afull_, i), 4); mbar_init(bar(aempty_, i), 1); }
        mbar_init(bar(&done_, 0), 1); mbar_init(bar(&tab_, 0), 1);
        mbar_fence_init();
    }
    if (tid < 8) s_total[tid] = 0ull;
    if (warp == 20) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "n"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    pdl_launch_dependents();
    const uint32_t tmem = tmem_base, items = ntiles * ns;      // an item: a segment of a tile
    bool ok = true;

    // copies: four threads a row and plane, 16 bytes each
    uint32_t l_item = 0, l_tile = 0, l_seg = 0, l_st = 0, l_ph = 1, l_n = ntiles ? tiles[0].n : 0u;
    const uint32_t ct = tid - PT_UNPACK, cpiece = ct & 3u, crow = ct >> 2;
    const uint64_t step32 = (uint64_t)32 * a.row_bytes;
    const uint8_t* l_src = ntiles ? tiles[0].base + (uint64_t)crow * a.row_bytes + s_lo * 64 + cpiece * 16 : nullptr;
    auto fetch = [&]() {
        const uint32_t dst = ring + l_st * G::STAGE + crow * G::PITCH + cpiece * 16;
        if ((s_lo + l_seg) * 64 + cpiece * 16 < a.plane) {
            const uint8_t* src = l_src;
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
                if (crow + 32 * k < l_n) {
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 32 * k * G::PITCH), "l"(src) : "memory");
                    if (PL == 2) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 32 * k * G::PITCH + 64), "l"(src + a.plane) : "memory");
                }
                src += step32;
            }
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar(full_, l_st)) : "memory");
        l_item++;
        l_src += 64;
        if (++l_st == a.stages) { l_st = 0; l_ph ^= 1u; }
        if (++l_seg == ns) {
            l_seg = 0; l_tile++;
            if (l_tile < ntiles) { l_n = tiles[l_tile].n; l_src = tiles[l_tile].base + (uint64_t)crow * a.row_bytes + s_lo * 64 + cpiece * 16; }
        }
    };
    const bool copies = warp >= PT_UNPACK / 32 && warp < (PT_UNPACK + PT_COPY) / 32;
    if (copies)
        for (uint32_t k = 0; k < a.stages && l_item < items; k++) fetch();

    pdl_wait();
    const uint32_t chunks = ns * 4 * G::CP;
    if (warp == 20 && lane == 0) {
        const uint32_t bytes = chunks * a.batch * 64;
        mbar_arrive_expect_tx(bar(&tab_, 0), bytes);
        bulk_g2s(ring + a.tab_off, a.table + (size_t)s_lo * 4 * G::CP * a.batch * 4, bytes, bar(&tab_, 0));
    }

    if (warp < 16) {               // ---- unpack: a group of four warps takes every fourth half of a segment, so the groups are at different work
        const uint32_t grp = warp >> 2, quad = warp & 3u;
        const uint32_t mine = tmem + grp * 2 * G::AW + ((quad * 32) << 16);
        uint32_t tile = 0, seg = grp >> 1, st = grp >> 1, ph = 0, aph = 1;
        while (st >= a.stages) st -= a.stages;
        while (seg >= ns) { seg -= ns; tile++; }
        for (uint32_t it = grp >> 1; it < items; it += 2) {
            const uint32_t n = tiles[tile].n;
            ok = warp_wait(bar(full_, st), ph, limit);
            if (!ok) break;
            const uint32_t at = ring + st * G::STAGE + (quad * 32 + lane) * G::PITCH + (grp & 1u) * 32;
            uint4 p[2], m[2];
#pragma unroll
            for (int h = 0; h < 2; h++) { p[h] = lds128(at + 16 * h); m[h] = PL == 2 ? lds128(at + 64 + 16 * h) : p[h]; }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(empty_, st));
            st += 2;
            if (st >= a.stages) { st -= a.stages; ph ^= 1u; }
            ok = warp_wait(bar(aempty_, grp), aph, limit);
            if (!ok) break;
            aph ^= 1u;
            if (32 * quad < n) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");      // the products that read the slot are done
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t pw[4] = {p[h].x, p[h].y, p[h].z, p[h].w}, mw[4] = {m[h].x, m[h].y, m[h].z, m[h].w};
                    uint32_t w[G::AW];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if constexpr (PL == 2) {
                            const PlaneFields two = plane_fields(pw[i], mw[i]);
                            const uint32_t even = even_fields(two), odd = odd_fields(two);
#pragma unroll
                            for (int k = 0; k < 4; k++) { w[8 * i + k] = field_bytes(even, k); w[8 * i + 4 + k] = field_bytes(odd, k); }
                        } else {
                            const uint32_t f = code_fields(pw[i]);
#pragma unroll
                            for (int k = 0; k < 4; k++) w[4 * i + k] = field_bytes(f, k);
                        }
                    }
                    if constexpr (PL == 2) tmem_put32(mine + h * G::AW, w); else tmem_put16(mine + h * G::AW, w);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            }
            if (lane == 0) mbar_arrive(bar(afull_, grp));
            seg += 2;
            while (seg >= ns) { seg -= ns; tile++; }
        }
    } else if (copies) {
        while (l_item < items) {
            ok = warp_wait(bar(empty_, l_st), l_ph, limit);
            if (!ok) break;
            fetch();
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (ok) ok = warp_wait(bar(&tab_, 0), 0, limit);
        if (ok) {
            const uint32_t cols4 = 4 * a.batch, each = PT_COPY / cols4, col = ct % cols4;      // a thread adds up chunks of one column of B
            long long sum = 0;
            if (ct < each * cols4)
                for (uint32_t c = ct / cols4; c < chunks; c += each) sum += field_total(*reinterpret_cast<const uint4*>(smem + a.tab_off + (c * cols4 + col) * 16));
            if (sum) atomicAdd(&s_total[col >> 2], (unsigned long long)(sum * digit_worth(col & 3u)));
        }
    } else {                       // ---- products
        constexpr uint32_t idesc = (2u << 4) | (1u << 10) | ((N / 8) << 17) | (8u << 24);      // u8 x s8 -> s32, 128 x N
        const uint32_t step = 2 * 64 * a.batch >> 4;      // descriptor units from product to product
        const uint32_t desc_hi = ((128u >> 4)) | (1u << 14), desc_lo = ((64 * a.batch) >> 4) << 16 | (((ring + a.tab_off) & 0x3FFFFu) >> 4);
        if (elect_lane()) {
            ok = mbar_wait_limit(bar(&tab_, 0), 0, limit);
            uint32_t half = 0, d = tmem + PT_D, lo = desc_lo;
            for (uint32_t j = 0; j < 2 * items && ok; j++) {
                const uint32_t g = j & 3u;
                ok = mbar_wait_limit(bar(afull_, g), (j >> 2) & 1u, limit);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t ta = tmem + g * 2 * G::AW, more = half > 0;
#pragma unroll
                for (uint32_t k = 0; k < G::CP; k++)
                    mma_u8s8_ta(d, ta + 8 * k, (uint64_t)desc_hi << 32 | (lo + k * step), idesc, k > 0 || more);
                mma_commit(bar(aempty_, g));
                lo += G::CP * step;
                if (++half == 2 * ns) { half = 0; d += N; lo = desc_lo; }
            }
            mma_commit(bar(&done_, 0));
            ok = mbar_wait_limit(bar(&done_, 0), 0, limit) && ok;
        }
        ok = __all_sync(0xffffffffu, ok);
    }
    if (!ok && lane == 0) atomicCAS(a.status, 0, KERR_PT_WAIT);
    __syncthreads();               // all products and copies are done: ring and table are free
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // [vector][row]: sums in fixed-point units, the digits of a sum meet in 64 bits
    auto* part = reinterpret_cast<long long*>(smem);
    const uint32_t VR = MATS * R;
    if (warp < 16) {
        const uint32_t quad = warp & 3u;
        for (uint32_t t = warp >> 2; t < ntiles; t += 4) {
            const uint32_t n = tiles[t].n;
            if (32 * quad >= n) continue;
            for (uint32_t v = 0; v < a.batch; v++) {
                uint32_t c[4];
                tmem_get4(c, tmem + PT_D + t * N + v * 4 + ((quad * 32) << 16));
                const long long s = ((long long)(int)c[0] * 128 + (int)c[1]) * 16384 + ((long long)(int)c[2] * 128 + (int)c[3]);
                if (32 * quad + lane < n) part[(size_t)v * VR + tiles[t].at + 32 * quad + lane] = s;
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    auto meet = [&]() {
        if (S > 1) {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else {
            __syncthreads();
        }
    };
    meet();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    for (uint32_t i = rank * PT_THREADS + tid; i < R * a.batch; i += S * PT_THREADS) {
        const uint32_t v = i / R, lr = i - v * R, gr = r_lo + lr;
        uint32_t s = 0;
        if (!SW) while (s + 1 < a.nw && gr >= a.row0[s + 1]) s++;
        const uint32_t row = gr - a.row0[s];
        const float kappa = __ldg(a.kappa + v);
        float f[MATS];
#pragma unroll
        for (uint32_t q = 0; q < MATS; q++) {
            const uint32_t at = v * VR + q * R + lr;
            long long sum = 0;
            if (S > 1) for (uint32_t r = 0; r < S; r++) sum += ld_cluster_s64(ring + at * 8, r) - ld_cluster_s64(smem_u32(s_total + v), r);
            else sum = part[at] - (long long)s_total[v];
            f[q] = kappa * (float)sum * __ldg((SW && q ? a.up_scale : a.scale[s]) + row);
        }
        float r = SW ? silu_ref(f[0]) * f[MATS - 1] : f[0];
        const uint32_t yi = a.y_off[s] + row;
        const size_t at = (size_t)v * a.y_stride + yi;
        if (a.resid != nullptr) r = __fadd_rn(__ldcg(a.resid + at), r);
        a.y[at] = r;
    }
    meet();                        // the others have read this CTA's sums
    if (warp == 20) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512));
}

template <int N, int PL, bool SW>
int plan_and_launch(PtArgs a, const LaunchCfg& cfg, bool dry, uint32_t* launches_out, float* us) {
    using G = PtGeom<PL>;
    constexpr uint32_t MATS = SW ? 2 : 1, MOST = std::min<uint32_t>(PT_TILES, (512 - PT_D) / N);
    static bool attr_done[64] = {};
    static int clusters[64][4] = {};
    auto kern = plane_tc_kernel<N, PL, SW>;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return ALICE_E_CUDA;
    if (!attr_done[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PT_SMEM) != cudaSuccess) return ALICE_E_CUDA;
        attr_done[dev] = true;
    }
    const uint32_t sms = (uint32_t)std::max(cfg.num_sms, 1), total = a.row0[a.nw];
    cudaLaunchConfig_t lc = {};
    lc.blockDim = dim3(PT_THREADS); lc.stream = cfg.stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    auto table_of = [&](uint32_t S) { return (size_t)((a.segs + S - 1) / S) * 4 * G::CP * a.batch * 64 + 256; };
    // Four CTAs to a cluster where the columns go that far (of 1, 2, 4 and 8, gate and up 28672 x 8192 of three vectors: -, 86, 64, 79 us, 8192 x 8192
    // of eight: -, 22.3, 14.1, 17.1), eight where their tables leave four no room for two stages.
    uint32_t best = 0, best_ncl = 0;
    for (uint32_t S = 1, l2 = 0; S <= 8 && S <= a.segs; S *= 2, l2++) {
        uint32_t ncl = sms;
        if (S > 1) {      // a cluster's CTAs sit in one GPC: what the chip holds at once is asked for, once per kernel and device
            int& known = clusters[dev][l2];
            if (!known) {
                at[0].val.clusterDim.x = S;
                lc.attrs = at; lc.numAttrs = 1; lc.gridDim = dim3(sms / S * S); lc.dynamicSmemBytes = PT_SMEM;
                int n = 0;
                if (sms < S || cudaOccupancyMaxActiveClusters(&n, kern, &lc) != cudaSuccess || n < 1) { cudaGetLastError(); break; }
                known = n;
            }
            ncl = std::min<uint32_t>((uint32_t)known, sms / S);
        }
        if (table_of(S) + 2 * G::STAGE > PT_SMEM) continue;
        best = S; best_ncl = std::min(ncl, total);
        if (S == 4) break;
    }
    if (!best) return ALICE_E_SHAPE;
    // accumulators of a launch's tiles stay in tensor memory: more rows take another launch
    const uint64_t most = (uint64_t)(MOST / MATS - (a.nw - 1)) * 128 * best_ncl;
    const uint32_t launches = (uint32_t)((total + most - 1) / most);
    if (launches_out) *launches_out = launches;
    if (us) {      // start of a launch; steps of 128 rows, full or not, and a segment; sums of a cluster's rows at its end
        constexpr float start = PL == 2 ? (N == 16 ? 7.1f : 8.2f) : N == 16 ? 6.8f : 7.2f, step = PL == 2 ? (N == 16 ? 0.54f : 0.63f) : N == 16 ? 0.38f : 0.43f;
        constexpr float sum = N == 16 ? 4.3e-4f : PL == 2 ? 2.4e-4f : 2.1e-4f;
        const uint32_t n = total / launches, per = (n + best_ncl - 1) / best_ncl;
        uint32_t tiles = 0;      // of the cluster that has most: rows of several matrices make more of them
        for (uint32_t c = 0; c < best_ncl; c++) {
            const uint32_t lo = (uint32_t)((uint64_t)n * c / best_ncl), hi = (uint32_t)((uint64_t)n * (c + 1) / best_ncl);
            uint32_t t = 0;
            for (uint32_t i = 0; i < a.nw; i++) {
                const uint32_t from = std::max(lo, a.row0[i]), to = std::min(hi, a.row0[i + 1]);
                if (from < to) t += (to - from + 127) / 128;
            }
            tiles = std::max(tiles, t);
        }
        *us = launches * (start + step * MATS * tiles * ((a.segs + best - 1) / best) + sum * MATS * per * a.batch) * (SW ? 0.9f : 1.0f);
    }
    if (dry) return ALICE_OK;
    a.stages = (uint32_t)std::min<size_t>(PT_STAGES, (PT_SMEM - table_of(best)) / G::STAGE);
    a.tab_off = a.stages * G::STAGE;
    const size_t smem = a.tab_off + table_of(best);
    at[0].val.clusterDim.x = best;
    lc.attrs = best > 1 ? at : at + 1;
    lc.numAttrs = (best > 1 ? 1 : 0) + (cfg.pdl ? 1 : 0);
    for (uint32_t l = 0; l < launches; l++) {
        a.row_lo = (uint32_t)((uint64_t)total * l / launches);
        a.nrows = (uint32_t)((uint64_t)total * (l + 1) / launches) - a.row_lo;
        const uint32_t ncl = std::min(best_ncl, a.nrows), per = (a.nrows + ncl - 1) / ncl;
        lc.gridDim = dim3(ncl * best); lc.dynamicSmemBytes = std::max<size_t>({smem, (size_t)MATS * per * a.batch * 8, PT_SMEM_MIN});
        if (cudaLaunchKernelEx(&lc, kern, a, best) != cudaSuccess) return ALICE_E_CUDA;
    }
    return ALICE_OK;
}

template <int PL>
int launch_n(const PtArgs& a, const LaunchCfg& cfg, bool dry, uint32_t* l, float* us) {
    if (a.up) return a.batch <= 4 ? plan_and_launch<16, PL, true>(a, cfg, dry, l, us) : plan_and_launch<32, PL, true>(a, cfg, dry, l, us);
    return a.batch <= 4 ? plan_and_launch<16, PL, false>(a, cfg, dry, l, us) : plan_and_launch<32, PL, false>(a, cfg, dry, l, us);
}

}  // namespace

int launch_planes_tc(const GemvOp& op, const LaunchCfg& cfg, bool dry, uint32_t* launches, float* us) {
    const WeightDesc& w0 = *op.w[0];
    const bool codes = w0.fmt == WF_SPARSE_TERNARY;
    if ((w0.fmt != WF_TERNARY && !codes) || op.npeers || op.norm_w || op.batch < 3 || op.batch > 8 || op.argmax_key) return ALICE_E_SHAPE;
    if (op.nw < 1 || op.nw > 3 || (op.up && op.nw != 1)) return ALICE_E_INVALID;
    PtArgs a = {};
    for (uint32_t i = 0; i < op.nw; i++) {
        const WeightDesc* w = op.w[i];
        if (!w || !w->data || !w->scales || !w->rows || ((uintptr_t)w->data & 15)) return ALICE_E_INVALID;
        if (w->fmt != w0.fmt || w->cols != w0.cols || w->row_bytes != w0.row_bytes) return ALICE_E_SHAPE;
        a.w[i] = w->data; a.scale[i] = w->scales; a.rows[i] = w->rows; a.y_off[i] = op.y_off[i];
        a.row0[i + 1] = a.row0[i] + w->rows;
    }
    if (op.up) {
        const WeightDesc& u = *op.up;
        if (u.fmt != w0.fmt || u.rows != w0.rows || u.cols != w0.cols || u.row_bytes != w0.row_bytes) return ALICE_E_SHAPE;
        if (!u.data || !u.scales || ((uintptr_t)u.data & 15)) return ALICE_E_INVALID;
        a.up = u.data; a.up_scale = u.scales;
    }
    if (!op.y || !op.x) return ALICE_E_INVALID;
    a.nw = op.nw;
    a.row_bytes = w0.row_bytes; a.plane = codes ? w0.row_bytes : w0.row_bytes / 2;
    if (a.plane % 16) return ALICE_E_SHAPE;         // rows begin on 16-byte boundaries
    a.segs = (a.plane + PLANE_SEG - 1) / PLANE_SEG;
    a.y = op.y; a.resid = op.resid; a.y_stride = op.y_stride ? op.y_stride : a.row0[op.nw]; a.batch = op.batch;
    a.status = cfg.status; a.wait_limit = op.wait_limit;
    const uint32_t chunks = a.segs * 4 * (codes ? PtGeom<1>::CP : PtGeom<2>::CP);
    const size_t table = (size_t)chunks * op.batch * 64;
    if (!dry) {
        if (!op.prep || ((uintptr_t)op.prep & 15) || table + 64 > op.prep_bytes) return ALICE_E_SHAPE;
        a.table = static_cast<const uint4*>(op.prep);
        a.kappa = reinterpret_cast<const float*>(static_cast<const uint8_t*>(op.prep) + table);
    }
    auto rows = [&](bool plan) { return codes ? launch_n<1>(a, cfg, plan, launches, us) : launch_n<2>(a, cfg, plan, launches, us); };
    int rc = rows(true);
    if (rc || dry) return rc;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((chunks + 255) / 256, op.batch); lc.blockDim = dim3(256); lc.stream = cfg.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at; lc.numAttrs = cfg.pdl ? 1 : 0;
    auto tk = codes ? plane_tc_table_kernel<1> : plane_tc_table_kernel<2>;
    if (cudaLaunchKernelEx(&lc, tk, op.x, w0.cols, op.batch, chunks, const_cast<uint4*>(a.table), const_cast<float*>(a.kappa)) != cudaSuccess) return ALICE_E_CUDA;
    return rows(false);
}

}  // namespace alice

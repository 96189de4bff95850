// Kernels and launch of csrc/gemv_planes.cuh.
#include <algorithm>

#include "../../include/alice_cuda.h"
#include "digits_dev.cuh"
#include "gemv_mma.cuh"
#include "gemv_planes.cuh"
#include "planes_dev.cuh"

namespace alice {
namespace {

constexpr uint32_t PLANE_SMEM = 220 * 1024;
constexpr uint32_t PLANE_HDR = 128;

// One thread's part of a digit table: word w of quad lane t in a 64-byte segment. Planes: bits 4 h .. 4 h + 3 of its four bytes; codes:
// the four code places of its four bytes (h = 0). out[digit] = the B words of the four.
template <bool CODES>
__device__ __forceinline__ void plane_digits(const float* x, uint32_t cols, bool vec4, const FixedScale to_fixed, uint32_t seg, uint32_t t, uint32_t w, uint32_t h, uint32_t (&out)[4][4]) {
#pragma unroll
    for (int d = 0; d < 4; d++) out[d][0] = out[d][1] = out[d][2] = out[d][3] = 0u;
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) {
        const uint32_t byte = seg * PLANE_SEG + t * 16 + w * 4 + i;
        const uint32_t e = CODES ? byte * 4 : byte * 8 + 4 * h;
        float xe[4] = {0.f, 0.f, 0.f, 0.f};
        if (vec4 && e < cols) {
            const float4 q = __ldcg(reinterpret_cast<const float4*>(x + e));
            xe[0] = q.x; xe[1] = q.y; xe[2] = q.z; xe[3] = q.w;
        } else {
#pragma unroll
            for (uint32_t k = 0; k < 4; k++)
                if (e + k < cols) xe[k] = __ldcg(x + e + k);
        }
#pragma unroll
        for (uint32_t jj = 0; jj < 4; jj++) {
            // what the consumer's A bytes are worth: 2^j for bits 0 .. 6, 2^6 for bit 7; 2^(2 q) for code place q
            const int sh = CODES ? (int)(2 * jj) : min((int)(4 * h + jj), 6);
            const int f = (to_units(xe[jj], to_fixed) + ((1 << sh) >> 1)) >> sh;
            uint8_t dg[193];          // digits land 64 apart
            mma_store_digits(dg, f);
#pragma unroll
            for (int d = 0; d < 4; d++) out[d][jj] |= (uint32_t)dg[64 * d] << (8 * i);
        }
    }
}

// Digit table of one vector per blockIdx.y (columns 4 (v & 1) .. + 3 of pair v >> 1); vectors past `batch` are zero columns. With
// RECS records of 512 bytes to a segment and pair: table[((seg * NT + pair) * RECS + record) * 32 + 4 * column + t].
template <bool CODES>
__global__ void __launch_bounds__(256) plane_table_kernel(const float* x, uint32_t cols, uint32_t batch, uint32_t segs, uint32_t nt, uint4* table, float* kappa_out) {
    __shared__ float red[8];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t v = blockIdx.y, tid = threadIdx.x;
    const float* xv = x + (size_t)min(v, batch - 1) * cols;
    const bool vec4 = can_vec4(xv, cols);
    bool finite;
    FixedScale to_fixed;
    float kappa;
    const float amax = vec_amax<256>(xv, cols, vec4, red, finite);
    fixed_scale<MMA_FIX_BITS>(amax, finite, to_fixed, kappa);
    if (blockIdx.x == 0 && tid == 0) kappa_out[v] = kappa;
    constexpr uint32_t RECS = CODES ? 4 : 8;
    const uint32_t i = blockIdx.x * 256 + tid, seg = i / (RECS * 4), t = i & 3u, wh = (i >> 2) % RECS;
    if (seg >= segs) return;
    uint32_t out[4][4];
    plane_digits<CODES>(xv, v < batch ? cols : 0u, vec4, to_fixed, seg, t, CODES ? wh : wh >> 1, CODES ? 0u : wh & 1u, out);
    uint4* rec = table + ((size_t)(seg * nt + (v >> 1)) * RECS + wh) * 32 + (v & 1u) * 16 + t;
#pragma unroll
    for (int d = 0; d < 4; d++) rec[d * 4] = make_uint4(out[d][0], out[d][1], out[d][2], out[d][3]);
}

__device__ __forceinline__ uint32_t word_of(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// 16 bytes of a row; a plane is a multiple of 4 bytes, of 16 with VEC16. Words past the plane are zero weights.
template <bool VEC16>
__device__ __forceinline__ uint4 plane_load(const uint8_t* p, uint32_t off, uint32_t plane) {
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (VEC16) {
        if (off < plane)
            asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p + off));
    } else {
        const uint32_t* q = reinterpret_cast<const uint32_t*>(p + off);
        if (off < plane) v.x = __ldg(q);
        if (off + 4 < plane) v.y = __ldg(q + 1);
        if (off + 8 < plane) v.z = __ldg(q + 2);
        if (off + 12 < plane) v.w = __ldg(q + 3);
    }
    return v;
}

// Which matrix and rows tile `tile` of the launch is (gate and up are two matrices of the same tiles).
struct PlaneTile { const uint8_t* a; const uint8_t* b; };
template <bool SW>
__device__ __forceinline__ PlaneTile plane_tile(const PlaneArgs& a, uint32_t tile, bool up, uint32_t g) {
    uint32_t s = 0;
    if (!SW) while (s + 1 < a.nw && tile >= a.tile0[s + 1]) s++;
    const uint8_t* w = SW && up ? a.up : a.w[s];
    const uint32_t r0 = (tile - a.tile0[s]) * 16, last = a.rows[s] - 1;   // rows past the last repeat it; their sums are not stored
    return {w + (size_t)min(r0 + g, last) * a.row_bytes, w + (size_t)min(r0 + g + 8, last) * a.row_bytes};
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A signed A word of four weights: those whose bit is set in p are worth 2^j, those in n -2^j (bits j .. 7 of their bytes set). A
// byte cannot be +2^7: bit 7 is moved to bit 6.
__device__ __forceinline__ uint32_t signed_planes(uint32_t p, uint32_t n, int j) {
    const int k = min(j, 6);
    const uint32_t m = 0x01010101u << k, x = (j == 7 ? n >> 1 : n) & m;
    return ((j == 7 ? p >> 1 : p) & m) | x * ((1u << (8 - k)) - 1u);
}
// Codes 00 = 0, 01 = +1, 11 = -1 at place q of four bytes, worth +-2^(2 q): the high bit is the sign.
__device__ __forceinline__ uint32_t signed_codes(uint32_t w, int q) {
    return (w & (0x01010101u << (2 * q))) | (w & (0x02020202u << (2 * q))) * ((1u << (7 - 2 * q)) - 1u);
}
__device__ __forceinline__ void mma_s8s8_acc(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: pairs of vectors. PL: bit planes of a row (2: pos | neg, 1: packed codes). S CTAs to a cluster.
template <int NT, int PL, bool SW, bool VEC16>
__global__ void __launch_bounds__(PLANE_WARPS * 32, 1) plane_rows_kernel(const __grid_constant__ PlaneArgs a, const uint32_t S) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float s_red[PLANE_WARPS], s_kappa[2];
    constexpr int MATS = SW ? 2 : 1;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3u;
    const uint32_t rank = S > 1 ? blockIdx.x % S : 0u, cl = blockIdx.x / S, ncl = gridDim.x / S;
    const uint32_t tiles = a.tile0[a.nw];
    const uint32_t t_lo = (uint32_t)((uint64_t)tiles * cl / ncl), nt_loc = (uint32_t)((uint64_t)tiles * (cl + 1) / ncl) - t_lo;
    const uint32_t s_lo = a.segs * rank / S, ns = a.segs * (rank + 1) / S - s_lo;
    const uint32_t bar = smem_u32(smem), tab = bar + PLANE_HDR;
    constexpr uint32_t SEGB = (PL == 2 ? 8u : 4u) * NT * 512u;        // table bytes of a segment
    auto* acc = reinterpret_cast<unsigned long long*>(smem + a.acc_off);   // [mat][tile][16 rows][2 NT]: two's complement sums in fixed-point units
    const uint32_t acc_n = MATS * a.tiles_max * 16 * NT * 2;
    if (tid == 0) { mbar_init(bar, 1); mbar_fence_init(); }
    for (uint32_t i = tid; i < acc_n; i += PLANE_WARPS * 32) acc[i] = 0ull;
    __syncthreads();
    pdl_launch_dependents();

    // this warp's share of the (tile, segment) pairs, gate tiles before up tiles
    const uint32_t items = MATS * nt_loc * ns;
    const uint32_t i_lo = items * warp / PLANE_WARPS, i_hi = items * (warp + 1) / PLANE_WARPS;
    // loader: runs PF items ahead of the products
    constexpr int PF = NT <= 2 ? 2 : 1;
    uint4 buf[PF + 1][PL][2];
    uint32_t l_item = i_lo, l_tile = ns ? i_lo / ns : 0u, l_seg = i_lo - l_tile * ns;
    PlaneTile lt{};
    if (i_lo < i_hi) lt = plane_tile<SW>(a, t_lo + (l_tile >= nt_loc ? l_tile - nt_loc : l_tile), l_tile >= nt_loc, g);
    auto load = [&](uint4 (&v)[PL][2]) {
        if (l_item >= i_hi) return;
        const uint32_t off = (s_lo + l_seg) * PLANE_SEG + t * 16;
#pragma unroll
        for (int p = 0; p < PL; p++) {
            v[p][0] = plane_load<VEC16>(lt.a + p * a.plane, off, a.plane);
            v[p][1] = plane_load<VEC16>(lt.b + p * a.plane, off, a.plane);
        }
        l_item++;
        if (++l_seg == ns) {
            l_seg = 0; l_tile++;
            if (l_item < i_hi) lt = plane_tile<SW>(a, t_lo + (l_tile >= nt_loc ? l_tile - nt_loc : l_tile), l_tile >= nt_loc, g);
        }
    };
#pragma unroll
    for (int k = 0; k < PF; k++) load(buf[k]);

    pdl_wait();
    bool ok = true;
    if constexpr (NT == 1) {
        // one or two vectors: every CTA makes the digits of its columns itself, which takes about as long as fetching them and saves
        // the launch of the table kernel in between. Columns of a second vector that is not there only reach its own sums.
        constexpr bool CODES = PL == 1;
        constexpr uint32_t RECS = CODES ? 4 : 8;
        for (uint32_t v = 0; v < a.batch; v++) {
            const float* xv = a.x + (size_t)v * a.cols;
            const bool vec4 = can_vec4(xv, a.cols);
            bool finite;
            FixedScale to_fixed;
            float kappa;
            const float amax = vec_amax<PLANE_WARPS * 32>(xv, a.cols, vec4, s_red, finite);
            fixed_scale<MMA_FIX_BITS>(amax, finite, to_fixed, kappa);
            if (tid == 0) s_kappa[v] = kappa;
            for (uint32_t i = tid; i < ns * RECS * 4; i += PLANE_WARPS * 32) {
                const uint32_t sl = i / (RECS * 4), wh = (i >> 2) % RECS;
                uint32_t out[4][4];
                plane_digits<CODES>(xv, a.cols, vec4, to_fixed, s_lo + sl, t, CODES ? wh : wh >> 1, CODES ? 0u : wh & 1u, out);
                uint4* rec = reinterpret_cast<uint4*>(smem + PLANE_HDR + sl * SEGB + wh * 512) + v * 16 + t;
#pragma unroll
                for (int d = 0; d < 4; d++) rec[d * 4] = make_uint4(out[d][0], out[d][1], out[d][2], out[d][3]);
            }
        }
        __syncthreads();
    } else {
        const uint32_t tab_bytes = ns * SEGB;
        if (tid == 0) {
            mbar_arrive_expect_tx(bar, tab_bytes);
            if (tab_bytes) bulk_g2s(tab, a.table + (size_t)s_lo * (SEGB / 16), tab_bytes, bar);
        }
        ok = mbar_wait_limit(bar, 0, a.wait_limit > 0 ? a.wait_limit : WAIT_CYCLE_LIMIT);
        if (!ok && lane == 0) atomicCAS(a.status, 0, KERR_WAIT_FULL);
    }

    int c[NT][4] = {};
    uint32_t tile = ns ? i_lo / ns : 0u, seg = i_lo - tile * ns;
    // the digits of a sum meet in 64 bits (a row of equal signs over equal activations leaves 32): lanes 2 k and 2 k + 1 have two each
    auto flush = [&]() {
        unsigned long long* row = acc + ((tile >= nt_loc ? a.tiles_max + (tile - nt_loc) : tile) * 16 + g) * (NT * 2) + (t >> 1);
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                long long v = (long long)c[n][2 * r] * 128 + c[n][2 * r + 1];
                const long long other = __shfl_xor_sync(0xffffffffu, v, 1);
                v = v * 16384 + other;
                if (!(t & 1u)) atomicAdd(row + r * 8 * (NT * 2) + n * 2, (unsigned long long)v);
                c[n][2 * r] = c[n][2 * r + 1] = 0;
            }
    };
    auto step = [&](const uint4 (&v)[PL][2]) {
        const uint8_t* rec = smem + PLANE_HDR + seg * SEGB + lane * 16;
        constexpr int H = PL == 2 ? 2 : 1;
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int h = 0; h < H; h++) {
                uint4 b0[NT], b1[NT];
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    b0[n] = *reinterpret_cast<const uint4*>(rec + (n * 4 * H + 2 * p * H + h) * 512);
                    b1[n] = *reinterpret_cast<const uint4*>(rec + (n * 4 * H + (2 * p + 1) * H + h) * 512);
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    uint32_t w[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int r = q & 1, i = 2 * p + (q >> 1);
                        w[q] = PL == 2 ? signed_planes(word_of(v[0][r], i), word_of(v[PL - 1][r], i), 4 * h + j) : signed_codes(word_of(v[0][r], i), j);
                    }
#pragma unroll
                    for (int n = 0; n < NT; n++) mma_s8s8_acc(c[n], w[0], w[1], w[2], w[3], word_of(b0[n], j), word_of(b1[n], j));
                }
            }
        if (++seg == ns) { flush(); seg = 0; tile++; }
    };
    if (ok) {
        uint32_t it = i_lo;
        while (it < i_hi) {
#pragma unroll
            for (int k = 0; k < PF + 1; k++) {
                if (it < i_hi) {
                    load(buf[(k + PF) % (PF + 1)]);
                    step(buf[k]);
                    it++;
                }
            }
        }
        if (seg != 0) flush();
    }
    if (S > 1) cluster_sync(); else __syncthreads();

    // sums of the cluster's CTAs, scale, epilogue: output (vector, row) pairs dealt to the CTAs of the cluster
    const uint32_t R = nt_loc * 16, outs = R * a.batch, first = rank * (PLANE_WARPS * 32);
    const uint32_t acc_s = smem_u32(acc);
    unsigned long long key = 0ull;
    for (uint32_t i = first + tid; ok && i < outs; i += S * (PLANE_WARPS * 32)) {
        const uint32_t v = i / R, lr = i - v * R, tl = t_lo + lr / 16;
        uint32_t s = 0;
        if (!SW) while (s + 1 < a.nw && tl >= a.tile0[s + 1]) s++;
        const uint32_t row = (tl - a.tile0[s]) * 16 + lr % 16;
        if (row >= a.rows[s]) continue;
        float f[MATS];
#pragma unroll
        for (int q = 0; q < MATS; q++) {
            const uint32_t at = acc_s + ((q * a.tiles_max * 16 + lr) * (NT * 2) + v) * 8;
            long long sum = 0;
            for (uint32_t r = 0; r < S; r++) sum += S > 1 ? ld_cluster_s64(at, r) : (long long)acc[(at - acc_s) / 8];
            f[q] = (NT == 1 ? s_kappa[v] : __ldg(a.kappa + v)) * (float)sum * __ldg((SW && q ? a.up_scale : a.scale[s]) + row);
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
    if (S > 1) cluster_sync();      // the others have read this CTA's sums
}

uint32_t log2u(uint32_t v) { uint32_t r = 0; while ((1u << (r + 1)) <= v) r++; return r; }

template <int NT, int PL, bool SW, bool VEC16>
int plan_and_launch(PlaneArgs a, const LaunchCfg& cfg, bool dry, float* us) {
    static int8_t attr_done[64] = {};
    static int clusters[64][4] = {};
    auto kern = plane_rows_kernel<NT, PL, SW, VEC16>;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return ALICE_E_CUDA;
    if (!attr_done[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PLANE_SMEM) != cudaSuccess) return ALICE_E_CUDA;
        // the weights come through L1: behind a kernel that had made nearly all of it shared memory (attention) a 70B layer took 8 us more
        if (cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 50) != cudaSuccess) return ALICE_E_CUDA;
        attr_done[dev] = 1;
    }
    const uint32_t sms = (uint32_t)std::max(cfg.num_sms, 1), tiles = a.tile0[a.nw];
    cudaLaunchConfig_t lc = {};
    lc.blockDim = dim3(PLANE_WARPS * 32);
    lc.stream = cfg.stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    for (uint32_t S = 1; S <= 8; S *= 2) {
        // a cluster's CTAs sit in one GPC: what the chip holds at once is asked for, once per kernel and device
        uint32_t ncl = sms;
        if (S > 1) {
            int& known = clusters[dev][log2u(S)];
            if (!known) {
                at[0].val.clusterDim.x = S;
                lc.attrs = at; lc.numAttrs = 1; lc.gridDim = dim3(sms / S * S); lc.dynamicSmemBytes = PLANE_SMEM;
                int n = 0;
                if (sms < S || cudaOccupancyMaxActiveClusters(&n, kern, &lc) != cudaSuccess || n < 1) { cudaGetLastError(); break; }
                known = n;
            }
            ncl = std::min<uint32_t>((uint32_t)known, sms / S);
        }
        ncl = std::min(ncl, tiles);
        const uint32_t per = (tiles + ncl - 1) / ncl, slice = (a.segs + S - 1) / S;
        const size_t table = (size_t)slice * NT * (PL == 2 ? 4096 : 2048), acc = (size_t)(SW ? 2 : 1) * per * 16 * NT * 16;
        const size_t smem = PLANE_HDR + table + acc;
        if (smem > PLANE_SMEM) continue;
        // fewer tiles than half the SMs: let more CTAs share a tile's columns
        if (S < 8 && tiles * S * 2 <= sms && a.segs >= 2 * S) continue;
        if (us) {      // start; steps of 16 rows and a segment that a warp makes; bytes of digits and of sums in shared memory
            constexpr float start = PL == 2 ? (NT < 4 ? 6.5f : 6.1f) : NT < 4 ? 5.3f : 6.1f, step = PL == 2 ? (NT < 4 ? 1.2f : 1.9f) : NT < 4 ? 0.57f : 1.0f;
            constexpr float digit = PL == 2 ? (NT < 4 ? 1.8e-5f : 2.6e-5f) : NT < 4 ? 2.2e-5f : 2.5e-5f, sum = NT < 4 ? (PL == 2 ? 1.30e-4f : 1.49e-4f) : PL == 2 ? 1.52e-4f : 1.43e-4f;
            *us = start + step * (SW ? 2 : 1) * per * slice / PLANE_WARPS + digit * table + sum * acc;
        }
        if (dry) return ALICE_OK;
        a.tiles_max = per;
        a.acc_off = (uint32_t)(PLANE_HDR + table);
        at[0].val.clusterDim.x = S;
        lc.gridDim = dim3(ncl * S); lc.dynamicSmemBytes = smem;
        lc.attrs = S > 1 ? at : at + 1;
        lc.numAttrs = (S > 1 ? 1 : 0) + (cfg.pdl ? 1 : 0);
        return cudaLaunchKernelEx(&lc, kern, a, S) == cudaSuccess ? ALICE_OK : ALICE_E_CUDA;
    }
    return ALICE_E_SHAPE;
}

template <int NT, int PL>
int launch_pl(const PlaneArgs& a, bool vec16, const LaunchCfg& cfg, bool dry, float* us) {
    if (a.up) return vec16 ? plan_and_launch<NT, PL, true, true>(a, cfg, dry, us) : plan_and_launch<NT, PL, true, false>(a, cfg, dry, us);
    return vec16 ? plan_and_launch<NT, PL, false, true>(a, cfg, dry, us) : plan_and_launch<NT, PL, false, false>(a, cfg, dry, us);
}
template <int NT>
int launch_nt(const PlaneArgs& a, bool codes, bool vec16, const LaunchCfg& cfg, bool dry, float* us) {
    return codes ? launch_pl<NT, 1>(a, vec16, cfg, dry, us) : launch_pl<NT, 2>(a, vec16, cfg, dry, us);
}
// pairs of vectors the kernels are built for
uint32_t plane_pairs(uint32_t batch) { return batch <= 2 ? 1u : batch <= 4 ? 2u : 4u; }

}  // namespace

size_t plane_prep_bytes(uint32_t cols, uint32_t batch) {
    return (size_t)((cols + 511) / 512) * plane_pairs(batch) * 4096 + 256 + 4096;   // codes: half the bytes for half the columns
}

int launch_planes(const GemvOp& op, const LaunchCfg& cfg, bool dry, uint32_t* launches, float* us) {
    if (launches) *launches = 1;
    const WeightDesc& w0 = *op.w[0];
    const bool codes = w0.fmt == WF_SPARSE_TERNARY;
    if ((w0.fmt != WF_TERNARY && !codes) || op.npeers || op.norm_w || op.batch == 0 || op.batch > 8 || (op.argmax_key && op.batch > 1)) return ALICE_E_SHAPE;
    if (op.nw < 1 || op.nw > 3 || (op.up && op.nw != 1)) return ALICE_E_INVALID;
    PlaneArgs a = {};
    uint32_t total = 0;
    bool vec16 = true;
    for (uint32_t i = 0; i < op.nw; i++) {
        const WeightDesc* w = op.w[i];
        if (!w || !w->data || !w->scales || !w->rows || ((uintptr_t)w->data & 15)) return ALICE_E_INVALID;
        if (w->fmt != w0.fmt || w->cols != w0.cols || w->row_bytes != w0.row_bytes) return ALICE_E_SHAPE;
        a.w[i] = w->data; a.scale[i] = w->scales; a.rows[i] = w->rows; a.y_off[i] = op.y_off[i];
        a.tile0[i + 1] = a.tile0[i] + (w->rows + 15) / 16;
        total += w->rows;
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
    vec16 = a.plane % 16 == 0;
    a.segs = (a.plane + PLANE_SEG - 1) / PLANE_SEG;
    const uint32_t nt = plane_pairs(op.batch);
    const size_t table = (size_t)a.segs * nt * (codes ? 2048 : 4096);
    a.y = op.y; a.resid = op.resid; a.y_stride = op.y_stride ? op.y_stride : total; a.batch = op.batch;
    a.argmax_key = op.argmax_key; a.status = cfg.status; a.wait_limit = op.wait_limit;
    a.x = op.x; a.cols = w0.cols;
    if (!dry && nt > 1) {
        if (!op.prep || ((uintptr_t)op.prep & 15) || table + 64 > op.prep_bytes) return ALICE_E_SHAPE;
        a.table = static_cast<const uint4*>(op.prep);
        a.kappa = reinterpret_cast<const float*>(static_cast<const uint8_t*>(op.prep) + table);
    }
    auto rows = [&](bool plan) { return nt == 1 ? launch_nt<1>(a, codes, vec16, cfg, plan, us) : nt == 2 ? launch_nt<2>(a, codes, vec16, cfg, plan, us) : launch_nt<4>(a, codes, vec16, cfg, plan, us); };
    int rc = rows(true);
    if (rc || dry) return rc;
    if (nt == 1) return rows(false);
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((a.segs + (codes ? 15 : 7)) / (codes ? 16 : 8), 2 * nt); lc.blockDim = dim3(256); lc.stream = cfg.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at; lc.numAttrs = cfg.pdl ? 1 : 0;
    auto tk = codes ? plane_table_kernel<true> : plane_table_kernel<false>;
    if (cudaLaunchKernelEx(&lc, tk, op.x, w0.cols, op.batch, a.segs, nt, const_cast<uint4*>(a.table), const_cast<float*>(a.kappa)) != cudaSuccess) return ALICE_E_CUDA;
    return rows(false);
}

}  // namespace alice

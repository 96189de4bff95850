// Kernel and launch of csrc/gemv_kq_rows.cuh.
//
// The tiles of csrc/gemv_kq_mma.cuh (16 rows of unpacked quants as A, the int8 activations of up to eight vectors as B, integer
// scales) fed by a ring per warp: 16 rows x one or two blocks a stage, cp.async, no barrier between warps. The activations of a
// CTA's columns stay in shared memory for the whole launch; a cluster of S CTAs shares the columns where those of all vectors fit
// no single CTA, or a matrix has few rows. The (tile, stage) pairs of a CTA are dealt evenly to its warps, the parts of a tile are
// added in a fixed order.
//
// What bounds it: HBM at the largest sizes (28672 x 8192 gate and up in Q4_K, four vectors: 52 us, 5.1 TB/s), else start and drain of the launch and,
// close behind, the ALU, which takes a bit operation every other clk (about 200 instructions per 16 rows x 256 columns of Q4_K, whatever the batch).
// Addresses of the copies made once a warp instead of for every piece: Q5_K 5003 x 2816, three vectors 8.5 -> 7.9 us, 28672 x 8192, eight
// vectors 55.0 -> 48.5; Q6_K 28672 x 8192, four 61.1 -> 55.4, 128256 x 4096, eight 121 -> 109.
#include <algorithm>

#include "../../include/alice_cuda.h"
#include "gemv_kq_mma.cuh"
#include "gemv_kq_rows.cuh"

namespace alice {
namespace {

constexpr int KR_WARPS = 16;
constexpr uint32_t KR_SMEM = 224 * 1024;

// blocks of a row in a stage, its 16-byte pieces, row pitch of a stage (64-bit reads of 4 rows x 32 bytes, or 32-bit reads of
// 8 rows x 16 bytes for Q6_K, fill the banks once), slack behind the activations of a vector for the same reason
template <int FMT> struct KrFmt;
template <> struct KrFmt<4> { using T = KqK4<false>; static constexpr uint32_t BB = 144, NB = 2, CH = 18, PITCH = 288, XPAD = 32, DG = 16; };
template <> struct KrFmt<5> { using T = KqK4<true>;  static constexpr uint32_t BB = 176, NB = 2, CH = 22, PITCH = 352, XPAD = 32, DG = 16; };
template <> struct KrFmt<6> { using T = KqQ6K;       static constexpr uint32_t BB = 210, NB = 1, CH = 14, PITCH = 240, XPAD = 16, DG = 32; };

struct KrArgs {
    const uint8_t* w[3];
    uint32_t rows[3], y_off[3], tile0[4], nw;
    const uint8_t* up;
    uint32_t row_bytes, nb;
    const int8_t* qs;            // [batch][nb * 256]
    const float* d;              // [batch][nb]
    const int16_t* bsums;        // [batch][nb][16]
    float* y;
    const float* resid;
    uint32_t y_stride, batch;
    uint32_t tile_lo, tiles;                                       // tiles of this launch
    uint32_t tiles_max, stages, acts_off, main_off, head_off;      // shared memory: rings | activations | main | head
};

// bytes of the activations of nb blocks: qs, d, digits
template <int FMT>
__host__ __device__ constexpr uint32_t kr_acts_bytes(uint32_t nb) { return 8u * (nb * 256u + KrFmt<FMT>::XPAD) + 8u * nb * 4u + 8u * nb * KrFmt<FMT>::DG; }

template <int FMT, bool SW>
__global__ void __launch_bounds__(KR_WARPS * 32, 1) kq_rows_kernel(const __grid_constant__ KrArgs a, const uint32_t S) {
    extern __shared__ __align__(128) uint8_t smem[];
    using F = KrFmt<FMT>;
    constexpr int MATS = SW ? 2 : 1;
    constexpr uint32_t CH = F::CH, STAGE = 16 * F::PITCH;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3u;
    const uint32_t rank = S > 1 ? blockIdx.x % S : 0u, cl = blockIdx.x / S, ncl = gridDim.x / S;
    const uint32_t t_own = (uint32_t)((uint64_t)a.tiles * cl / ncl), nt_loc = (uint32_t)((uint64_t)a.tiles * (cl + 1) / ncl) - t_own;
    const uint32_t t_lo = a.tile_lo + t_own;
    const uint32_t all = (a.nb + F::NB - 1) / F::NB, s_lo = all * rank / S, ns = all * (rank + 1) / S - s_lo;
    const uint32_t b_lo = s_lo * F::NB, b_hi = min(a.nb, (s_lo + ns) * F::NB), nblk = b_hi - b_lo;
    const uint32_t base = smem_u32(smem), ring = base + warp * a.stages * STAGE;
    float* mainp = reinterpret_cast<float*>(smem + a.main_off);     // [mat][tile][16 rows][8]
    float* head = reinterpret_cast<float*>(smem + a.head_off);      // [warp][16 rows][8]
    pdl_launch_dependents();

    const uint32_t items = MATS * nt_loc * ns;
    const uint32_t i_lo = items * warp / KR_WARPS, i_hi = items * (warp + 1) / KR_WARPS;
    auto matrix_of = [&](uint32_t tile, uint32_t& s, const uint8_t*& w, uint32_t& r0) {     // tile: gate tiles, then up tiles
        const bool up = SW && tile >= nt_loc;
        const uint32_t tl = t_lo + (up ? tile - nt_loc : tile);
        s = 0;
        if (!SW) while (s + 1 < a.nw && tl >= a.tile0[s + 1]) s++;
        w = up ? a.up : a.w[s];
        r0 = (tl - a.tile0[s]) * 16;
    };
    // Where this lane's 16-byte pieces of a stage lie relative to the tile and the slot: the same for all tiles but a matrix's last one, so a
    // piece costs an addition and the copy (with the addresses made anew each time, 14 instructions, a quarter of the kernel's).
    constexpr uint32_t PIECES = (16 * CH + 31) / 32;
    uint32_t rel[PIECES];
#pragma unroll
    for (uint32_t j = 0; j < PIECES; j++) {
        const uint32_t i = j * 32 + lane, r = i / CH;
        rel[j] = r * a.row_bytes + (FMT == 6 ? 0u : (i - r * CH) * 16);
    }
    const uint32_t inside = 16 + (CH * 16 + a.row_bytes - 1) / a.row_bytes;      // rows from a tile's first one on that its whole stages may touch
    uint32_t l_item = i_lo, l_tile = i_lo / ns, l_seg = i_lo - l_tile * ns, l_slot = 0;
    const uint8_t *lw = nullptr, *lp = nullptr;      // matrix; this stage's columns of the tile's first row
    uint32_t ls = 0, lr0 = 0;
    auto to_tile = [&]() {
        matrix_of(l_tile, ls, lw, lr0);
        lp = lw + (uint64_t)lr0 * a.row_bytes + (uint64_t)(s_lo + l_seg) * (F::NB * F::BB);
    };
    if (i_lo < i_hi) to_tile();
    auto fetch = [&]() {
        if (l_item < i_hi) {
            const uint32_t dst = ring + l_slot * STAGE;
            if (lr0 + inside <= a.rows[ls]) {
#pragma unroll
                for (uint32_t j = 0; j < PIECES; j++) {
                    const uint32_t i = j * 32 + lane;
                    if (16 * CH % 32 && i >= 16 * CH) continue;
                    if constexpr (FMT != 6) {
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 16), "l"(lp + rel[j]) : "memory");
                    } else {
                        const uint32_t r = i / CH, c = i - r * CH;
                        const uint8_t* q = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(lp + rel[j]) & ~(uintptr_t)15);
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + r * F::PITCH + c * 16), "l"(q + c * 16) : "memory");
                    }
                }
            } else {        // rows past the last repeat it, nothing past the matrix is read
                const uint64_t total = (uint64_t)a.rows[ls] * a.row_bytes;
                const uint32_t at = (s_lo + l_seg) * (F::NB * F::BB);
                // Unrolled for Q6_K, though hardly ever run: the compiler then schedules the other path better (28672 x 8192, four vectors 63.9 us as a loop, 55.4
                // unrolled; 61.1 with no other path). Of Q4_K and Q5_K it is the loop (4096 x 4096, eight vectors 7.0 and 8.3 us).
#pragma unroll (FMT == 6 ? PIECES : 1)
                for (uint32_t i = lane; i < 16 * CH; i += 32) {
                    const uint32_t r = i / CH, c = i - r * CH;
                    const uint64_t off = (((uint64_t)min(lr0 + r, a.rows[ls] - 1) * a.row_bytes + at) & ~(uint64_t)15) + c * 16;
                    const uint32_t n = off < total ? (uint32_t)min((uint64_t)16, total - off) : 0u;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + r * F::PITCH + c * 16), "l"(n ? lw + off : lw), "r"(n) : "memory");
                }
            }
            l_item++;
            lp += F::NB * F::BB;
            if (++l_seg == ns) { l_seg = 0; l_tile++; if (l_item < i_hi) to_tile(); }
            if (++l_slot == a.stages) l_slot = 0;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (uint32_t k = 0; k + 1 < a.stages; k++) fetch();

    pdl_wait();
    // activations of this CTA's columns; columns of vectors past the batch stay as they are (a column only reaches its own results)
    uint8_t* const area = smem + a.acts_off;
    const uint32_t xs = nblk * 256 + F::XPAD;
    float* const xd = reinterpret_cast<float*>(area + 8u * xs);
    uint8_t* const xg = reinterpret_cast<uint8_t*>(xd + 8u * nblk);
    for (uint32_t i = tid; i < a.batch * nblk * 16; i += KR_WARPS * 32) {
        const uint32_t v = i / (nblk * 16), j = i - v * (nblk * 16);
        *reinterpret_cast<uint4*>(area + v * xs + j * 16) = __ldcg(reinterpret_cast<const uint4*>(a.qs + ((size_t)v * a.nb + b_lo) * 256 + j * 16));
    }
    for (uint32_t i = tid; i < a.batch * nblk; i += KR_WARPS * 32) {
        const uint32_t v = i / nblk, b = i - v * nblk;
        const size_t at = (size_t)v * a.nb + b_lo + b;
        xd[v * nblk + b] = __ldcg(a.d + at);
        const uint4 s0 = __ldcg(reinterpret_cast<const uint4*>(a.bsums + at * 16)), s1 = __ldcg(reinterpret_cast<const uint4*>(a.bsums + at * 16) + 1);
        kq_store_digits<FMT == 6>(smem_u32(xg + (v * nblk + b) * F::DG), s0, s1);
    }
    KqActs x;
    x.qs = smem_u32(area); x.xs = xs; x.d = smem_u32(xd); x.bsd = x.bs16 = smem_u32(xg); x.nb = nblk;
    __syncthreads();

    float acc[4] = {};           // rows g and g + 8, vectors 2 t and 2 t + 1
    uint32_t tile = i_lo / ns, seg = i_lo - tile * ns, slot = 0;
    bool mid = seg != 0;                     // this warp took the tile up in its middle
    uint32_t offA = 0, offB = 0;             // where the rows begin, modulo 16 (Q6_K blocks start anywhere)
    auto rows_of = [&]() {
        if (FMT != 6) return;
        uint32_t s, r0;
        const uint8_t* w;
        matrix_of(tile, s, w, r0);
        offA = min(r0 + g, a.rows[s] - 1) * a.row_bytes;
        offB = min(r0 + g + 8, a.rows[s] - 1) * a.row_bytes;
    };
    if (i_lo < i_hi) rows_of();
    auto flush = [&]() {
        float* dst = mid ? head + warp * 128 : mainp + (size_t)((tile >= nt_loc ? a.tiles_max + (tile - nt_loc) : tile) * 128);
        *reinterpret_cast<float2*>(dst + g * 8 + 2 * t) = make_float2(acc[0], acc[1]);
        *reinterpret_cast<float2*>(dst + (g + 8) * 8 + 2 * t) = make_float2(acc[2], acc[3]);
        acc[0] = acc[1] = acc[2] = acc[3] = 0.0f;
        mid = false;
    };
    for (uint32_t it = i_lo; it < i_hi; it++) {
        if (a.stages == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
        else if (a.stages == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 2;" ::: "memory");
        __syncwarp();                        // the stage is in for every lane, and every lane is done with the one before
        fetch();
        const uint32_t b0 = seg * F::NB, b1 = min(nblk, b0 + F::NB), at = (b_lo + b0) * F::BB;
        uint32_t rowA = ring + slot * STAGE + g * F::PITCH, rowB = rowA + 8 * F::PITCH;
        if (FMT == 6) { rowA += (offA + at) & 15u; rowB += (offB + at) & 15u; }
        if (++slot == a.stages) slot = 0;
        F::T::tile(rowA - b0 * F::BB, rowB - b0 * F::BB, b0, b1, x, lane, acc);
        if (++seg == ns) { flush(); seg = 0; tile++; if (it + 1 < i_hi) rows_of(); }
    }
    if (seg != 0 && i_lo < i_hi) flush();
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // parts of tiles that another warp began, in the order of the warps
    if (tid < 128) {
        for (uint32_t w = 1; w < (uint32_t)KR_WARPS; w++) {
            const uint32_t lo = items * w / KR_WARPS, hi = items * (w + 1) / KR_WARPS, tl = lo / ns;
            if (lo < hi && lo != tl * ns) mainp[(size_t)(tl >= nt_loc ? a.tiles_max + (tl - nt_loc) : tl) * 128 + tid] += head[w * 128 + tid];
        }
    }
    if (S > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
    const uint32_t R = nt_loc * 16, outs = R * a.batch;
    const uint32_t main_s = base + a.main_off;
    for (uint32_t i = rank * (KR_WARPS * 32) + tid; i < outs; i += S * (KR_WARPS * 32)) {
        const uint32_t v = i / R, lr = i - v * R, tl = t_lo + lr / 16;
        uint32_t s = 0;
        if (!SW) while (s + 1 < a.nw && tl >= a.tile0[s + 1]) s++;
        const uint32_t row = (tl - a.tile0[s]) * 16 + lr % 16;
        if (row >= a.rows[s]) continue;
        float f[MATS];
#pragma unroll
        for (int q = 0; q < MATS; q++) {
            const uint32_t at = main_s + ((q * a.tiles_max * 16 + lr) * 8 + v) * 4;
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
            f[q] = y;
        }
        float r = SW ? silu_ref(f[0]) * f[MATS - 1] : f[0];
        const size_t at = (size_t)v * a.y_stride + a.y_off[s] + row;
        if (a.resid != nullptr) r = __fadd_rn(__ldcg(a.resid + at), r);
        a.y[at] = r;
    }
    if (S > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

template <int FMT, bool SW>
int plan_and_launch(KrArgs a, const LaunchCfg& cfg, bool dry, uint32_t* launches_out) {
    using F = KrFmt<FMT>;
    static bool attr_done[64] = {};
    static int clusters[64][4] = {};
    auto kern = kq_rows_kernel<FMT, SW>;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return ALICE_E_CUDA;
    if (!attr_done[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)KR_SMEM) != cudaSuccess) return ALICE_E_CUDA;
        attr_done[dev] = true;
    }
    const uint32_t sms = (uint32_t)std::max(cfg.num_sms, 1), tiles = a.tile0[a.nw], all = (a.nb + F::NB - 1) / F::NB;
    cudaLaunchConfig_t lc = {};
    lc.blockDim = dim3(KR_WARPS * 32); lc.stream = cfg.stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    // The smallest cluster whose CTAs hold the activations of their columns and the sums of all their tiles. Where none does (large matrices:
    // Q5_K from some 25000 x 8192 on), the one that takes the fewest launches, each over a part of the rows: 28672 x 8192 in Q5_K 57 us
    // for eight vectors, 261 one vector at a time.
    constexpr size_t TILE = (size_t)(SW ? 2 : 1) * 16 * 8 * 4, HEAD = (size_t)KR_WARPS * 16 * 8 * 4, STAGE = (size_t)KR_WARPS * 16 * F::PITCH;
    auto acts_of = [&](uint32_t S) { return (kr_acts_bytes<FMT>((all + S - 1) / S * F::NB) + 15u) & ~(size_t)15; };
    uint32_t best = 0, best_ncl = 0, launches = 0;
    for (uint32_t S = 1, l2 = 0; S <= 8 && S <= all && launches != 1; S *= 2, l2++) {
        uint32_t ncl = sms;
        if (S > 1) {      // a cluster's CTAs sit in one GPC: what the chip holds at once is asked for, once per kernel and device
            int& known = clusters[dev][l2];
            if (!known) {
                at[0].val.clusterDim.x = S;
                lc.attrs = at; lc.numAttrs = 1; lc.gridDim = dim3(sms / S * S); lc.dynamicSmemBytes = KR_SMEM;
                int n = 0;
                if (sms < S || cudaOccupancyMaxActiveClusters(&n, kern, &lc) != cudaSuccess || n < 1) { cudaGetLastError(); break; }
                known = n;
            }
            ncl = std::min<uint32_t>((uint32_t)known, sms / S);
        }
        ncl = std::min(ncl, tiles);
        const size_t fixed = acts_of(S) + HEAD + 2 * STAGE;
        if (fixed + TILE > KR_SMEM) continue;
        // fewer tiles than half the SMs: let more CTAs share a tile's columns
        if (S < 8 && tiles * S * 2 <= sms && all >= 2 * S) continue;
        const uint64_t room = (uint64_t)ncl * ((KR_SMEM - fixed) / TILE);      // tiles of a launch
        const uint32_t need = (uint32_t)((tiles + room - 1) / room);
        if (!best || need < launches) { best = S; best_ncl = ncl; launches = need; }
    }
    if (!best) return ALICE_E_SHAPE;
    if (launches_out) *launches_out = launches;
    if (dry) return ALICE_OK;
    const size_t acts = acts_of(best);
    at[0].val.clusterDim.x = best;
    lc.attrs = best > 1 ? at : at + 1;
    lc.numAttrs = (best > 1 ? 1 : 0) + (cfg.pdl ? 1 : 0);
    for (uint32_t l = 0; l < launches; l++) {
        a.tile_lo = (uint32_t)((uint64_t)tiles * l / launches);
        a.tiles = (uint32_t)((uint64_t)tiles * (l + 1) / launches) - a.tile_lo;
        const uint32_t ncl = std::min(best_ncl, a.tiles);
        a.tiles_max = (a.tiles + ncl - 1) / ncl;
        const size_t mn = a.tiles_max * TILE, fixed = acts + mn + HEAD;
        a.stages = (uint32_t)std::min<size_t>(4, (KR_SMEM - fixed) / STAGE);
        a.acts_off = (uint32_t)(a.stages * STAGE); a.main_off = (uint32_t)(a.acts_off + acts); a.head_off = (uint32_t)(a.main_off + mn);
        lc.gridDim = dim3(ncl * best); lc.dynamicSmemBytes = fixed + a.stages * STAGE;
        if (cudaLaunchKernelEx(&lc, kern, a, best) != cudaSuccess) return ALICE_E_CUDA;
    }
    return ALICE_OK;
}

}  // namespace

int launch_kq_rows(const GemvOp& op, const LaunchCfg& cfg, bool dry, uint32_t* launches) {
    const WeightDesc& w0 = *op.w[0];
    const bool q4 = w0.fmt == WF_Q4_K, q5 = w0.fmt == WF_Q5_K;
    if ((!q4 && !q5 && w0.fmt != WF_Q6_K) || !op.q8 || op.npeers || op.norm_w || op.batch == 0 || op.batch > 8 || op.argmax_key) return ALICE_E_SHAPE;
    if (op.nw < 1 || op.nw > 3 || (op.up && op.nw != 1) || !op.y || w0.cols % 256 || !w0.cols || op.q8->nb * 256 != w0.cols) return ALICE_E_SHAPE;
    if (!op.q8->qs || ((uintptr_t)op.q8->qs & 15) || ((uintptr_t)op.q8->bsums & 15)) return ALICE_E_SHAPE;
    KrArgs a = {};
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
    a.nw = op.nw; a.row_bytes = w0.row_bytes; a.nb = w0.cols / 256;
    a.qs = op.q8->qs; a.d = op.q8->d; a.bsums = op.q8->bsums;
    a.y = op.y; a.resid = op.resid; a.y_stride = op.y_stride ? op.y_stride : total; a.batch = op.batch;
    if (op.up) return q4 ? plan_and_launch<4, true>(a, cfg, dry, launches) : q5 ? plan_and_launch<5, true>(a, cfg, dry, launches) : plan_and_launch<6, true>(a, cfg, dry, launches);
    return q4 ? plan_and_launch<4, false>(a, cfg, dry, launches) : q5 ? plan_and_launch<5, false>(a, cfg, dry, launches) : plan_and_launch<6, false>(a, cfg, dry, launches);
}

}  // namespace alice

// Matvec over ternary bit planes and packed ternary codes for 1..8 input vectors in ONE pass over the weights.
//
// The weights are the A operand of the int8 mma.sync and the fixed-point digits of the activations the B operand, as in
// csrc/gemv_mma.cuh, but the bytes go from HBM straight into the fragment registers: lane (g, t) of a warp loads 16 bytes of rows
// g and g + 8 at byte 16 t of a 64-byte segment, which is a whole A fragment for any order of the columns that the B side shares.
// No ring, no barrier per stage, no shared-memory read of a weight. Three operations turn the two planes' bits j (or one code
// place) of four weights into a signed byte each, +-2^j, so a weight takes part in one product, not two. The digits of two
// vectors fill the eight B columns, so a second vector costs nothing and every further pair costs its products only: 8 clk
// per m16n8k32 and SM quarter, measured.
//
// 28672 x 8192: one vector 20.0 us (27.8 by the ring kernel). What bounds it: the stream and the instructions on it alike (2.9 TB/s). Three vectors
// and more go to csrc/gemv_planes_tc.cu where that is the faster (eight: 37.5 us here, 24.5 there).
//
// Split: a cluster of S CTAs owns a range of 16-row tiles, each of its CTAs 1 / S of the columns, whose digit table stays in
// shared memory for the whole launch (S is the smallest that makes it fit, or larger where a matrix has fewer tiles than the
// chip has SMs). Inside a CTA the (tile, segment) pairs are dealt evenly to 16 warps; sums are integers, added in shared memory
// with atomics (exact, so the order does not matter) and once per launch over the cluster.
#pragma once
#include "gemv_launch.cuh"

namespace alice {

constexpr uint32_t PLANE_SEG = 64;                      // bytes of a plane one step covers
constexpr int PLANE_WARPS = 16;

struct PlaneArgs {
    const uint8_t* w[3];
    const float* scale[3];
    uint32_t rows[3], y_off[3], tile0[4];               // tiles of matrix i: [tile0[i], tile0[i + 1])
    uint32_t nw;
    const uint8_t* up;                                  // fused SwiGLU: w[0] = gate
    const float* up_scale;
    uint32_t row_bytes, plane, segs;                    // bytes of a row and of a plane; 64-byte segments of a plane
    const float* x;                                     // one or two vectors: the kernel makes the digits itself
    uint32_t cols;
    const uint4* table;                                 // more: see plane_table_kernel
    const float* kappa;                                 // value of one fixed-point unit, per vector
    float* y;
    const float* resid;
    uint32_t y_stride, batch;
    unsigned long long* argmax_key;                     // batch 1 only
    uint32_t tiles_max;                                 // most tiles a cluster owns
    uint32_t acc_off;                                   // shared memory: barrier | table slice | sums
    int* status;
    long long wait_limit;
};

// Rows (planes of rows) that begin on 16-byte boundaries.
inline bool plane_rows_aligned(const WeightDesc& w) { return (w.fmt == WF_SPARSE_TERNARY ? w.row_bytes : w.row_bytes / 2) % 16 == 0; }
// Scratch for the digit table of `batch` vectors, for either format.
size_t plane_prep_bytes(uint32_t cols, uint32_t batch);
// ALICE_E_SHAPE: not a case for this kernel (the caller goes on to the ring kernels). dry: plan only. launches: of the product, which is one. us: about what
// three vectors and more take, tables included.
int launch_planes(const GemvOp& op, const LaunchCfg& cfg, bool dry, uint32_t* launches = nullptr, float* us = nullptr);
// The same for three vectors and more on tcgen05, where plane_rows_aligned.
int launch_planes_tc(const GemvOp& op, const LaunchCfg& cfg, bool dry, uint32_t* launches = nullptr, float* us = nullptr);

}  // namespace alice

// Matvec over Q8_0, Q1_0 and Q2_0 blocks for 1..8 input vectors in ONE pass over the weights.
#pragma once
#include "gemv_launch.cuh"

namespace alice {

// Scratch for the digit table of `batch` vectors, Q1_0 or Q2_0 (Q8_0 needs none).
size_t blocks_prep_bytes(uint32_t cols, uint32_t batch);
// ALICE_E_SHAPE: not a case for this kernel (the caller goes on to the ring kernels). dry: plan only. launches: of the product, which is one.
int launch_blocks(const GemvOp& op, const LaunchCfg& cfg, bool dry, uint32_t* launches = nullptr);

}  // namespace alice

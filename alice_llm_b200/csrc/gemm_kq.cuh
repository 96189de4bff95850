// Products of K-quant matrices with many vectors (the tokens of a prompt): weights unpacked once per tile of tokens.
#pragma once
#include "gemv_launch.cuh"

namespace alice {

// Any number of vectors in op.batch with op.q8 prepared. ALICE_E_SHAPE: not a case for this kernel. dry: plan only.
int launch_kq_gemm(const GemvOp& op, const LaunchCfg& cfg, bool dry);

}  // namespace alice

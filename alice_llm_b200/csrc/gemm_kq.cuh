// Products of K-quant matrices with many vectors (the tokens of a prompt): weights unpacked once per tile of tokens.
#pragma once
#include "gemv_launch.cuh"

namespace alice {

// Any number of vectors in op.batch with op.q8 prepared. ALICE_E_SHAPE: not a case for this kernel.
int launch_kq_gemm(const GemvOp& op, const LaunchCfg& cfg);

// The same for more than 64 vectors of operands launch_kq_gemm has checked (csrc/gemm_kq_tc.cu), with kq_tc_prep_bytes of scratch in
// op.prep; ALICE_E_SHAPE without it.
int launch_kq_gemm_tc(const GemvOp& op, const LaunchCfg& cfg);
size_t kq_tc_prep_bytes(uint32_t cols, uint32_t batch);

}  // namespace alice

// Matvec over K-quant rows for up to 8 Q8_K vectors in ONE pass over the weights, on the int8 tensor path.
#pragma once
#include "gemv_launch.cuh"

namespace alice {

// ALICE_E_SHAPE: not a case for this kernel. dry: plan only. launches: how many this takes.
int launch_kq_rows(const GemvOp& op, const LaunchCfg& cfg, bool dry, uint32_t* launches = nullptr);

}  // namespace alice

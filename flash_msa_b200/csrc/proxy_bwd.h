// Proxy half of the fused backward (proxy_bwd.cu), launched by fmsa_sparse_bwd behind the main kernel.
#pragma once

#include <cuda_runtime.h>

#include "../../include/flash_msa_b200.h"
#include "msa_common.cuh"

namespace fmsa {

// `teacher_dqp`: on entry the teacher of every edge of the pass (written by the main kernel), on return dQp partial rows.  units.counter has been zeroed.
int launch_proxy_bwd(const fmsa_problem* pb, const fmsa_tensor& q_proxy, const fmsa_tensor& k_proxy, const float* lse_proxy,
                     const UnitSpace& units, const int32_t* col_q, void* teacher_dqp, int64_t part_slots, int split,
                     float* dkp_acc, float* kl_value, int grid, int32_t* status, cudaStream_t stream);

}  // namespace fmsa

// Proxy half of the fused backward (proxy_bwd.cu), launched by fmsa_sparse_bwd behind the main kernel.
#pragma once

#include <cuda_runtime.h>

#include "../../include/flash_msa_b200.h"
#include "msa_common.cuh"

namespace fmsa {

// The teacher of a chunk of 128 gathered rows: from its first row's slot on, 8 rows are 2048 bytes [key][4] of fp16 pairs (rows 2i and
// 2i + 1 of the eight in word i), so that a thread, which has one key, moves 16 bytes at a time; of a last group of fewer rows every pair
// is 512 bytes [key] of such words and an odd last row 256 bytes [key].  (With all pairs as 512 bytes [key] and 4-byte accesses the backward
// kernels took 1.526 instead of 1.519 ms at B=2 S=8192 Hq=32 top-k 16 blocks, 1.680 instead of 1.668 dense at B=4 S=4096, 3.507 instead of
// 3.448 at B=1 S=65536 top-k 32, the prefetch of positions in proxy_bwd.cu included.)
// `teacher_dqp`: on entry the teacher of every edge of the pass (written by the main kernel), on return dQp partial rows.  units.counter has been zeroed.
int launch_proxy_bwd(const fmsa_problem* pb, const fmsa_tensor& q_proxy, const fmsa_tensor& k_proxy, const float* lse_proxy,
                     const UnitSpace& units, const int32_t* col_q, void* teacher_dqp, int64_t part_slots, int split,
                     float* dkp_acc, float* kl_value, int grid, int32_t* status, cudaStream_t stream);

}  // namespace fmsa

// Launchers shared by the C-ABI entry points of single stages and the whole-pass entry points (pipeline.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/flash_msa_b200.h"

namespace fmsa {

// Rows of query tiles first_tile .. of the reverse index; `row_start`: where they begin in its rows (first_tile > 0).
// `counter`: one zeroed word.
int launch_sparse_fwd(const fmsa_problem* pb, const fmsa_tensor* q, const fmsa_tensor* k, const fmsa_tensor* v,
                      const fmsa_tensor* q_proxy, const fmsa_tensor* k_proxy, const int32_t* row_ptr,
                      const int32_t* row_start, int first_tile, const int32_t* col_q, void* o_part, float* lse_part, int64_t part_slots, int g_begin, int g_count, int with_proxy, int dense,
                      int32_t* counter, int32_t* status, cudaStream_t st);
// `sinks`: fp32 [Hq] softmax-bias logits or null.
int launch_fwd_combine(const fmsa_problem* pb, const void* o_part, const float* lse_part, const int32_t* edge_pos,
                       const int32_t* row_ptr, void* out, float* lse, float* lse_proxy, const float* sinks, int first_tile, int g_begin, int g_count, int dense, cudaStream_t st);
// Query tiles 0 .. tiles-1 of every (batch, proxy head).  `visits`: from select_fused_launch, or where the selection is another one from
// reverse_index_launch or launch_tile_visits (null if dense); lse_proxy null: without the proxy head.  `counter`: one zeroed word.  One
// launch, and one more with sinks.
int launch_tile_fwd(const fmsa_problem* pb, const fmsa_tensor* q, const fmsa_tensor* k, const fmsa_tensor* v, const fmsa_tensor* q_proxy,
                    const fmsa_tensor* k_proxy, const void* visits, void* out, float* lse, float* lse_proxy, const float* sinks, float* zero,
                    int tiles, int dense, int32_t* counter, int32_t* status, cudaStream_t st);
// `counter`, `counter_proxy`: zeroed here if `zero_counters` (they may then be the same word).
int launch_sparse_bwd(const fmsa_problem* pb, const fmsa_tensor* q, const fmsa_tensor* k, const fmsa_tensor* v,
                      const fmsa_tensor* q_proxy, const fmsa_tensor* k_proxy, const fmsa_tensor* d_out, const float* lse,
                      const float* lse_proxy, const float* delta, const int32_t* row_ptr, const int32_t* col_q, void* dq_part,
                      void* dqp_part, int64_t part_slots, int split, float* dkp_acc, float* dk_acc, float* dv_acc, int g_begin,
                      int g_count, int with_kl, int dense, float* kl_value, int32_t* counter, int32_t* counter_proxy,
                      bool zero_counters, int32_t* status, cudaStream_t st);

// One (B,H,S,128) gradient from its contiguous fp32 accumulator: dst = 16-bit (src * scale * (*factor or 1)).
struct CastJob {
    const float* src;
    void* dst;
    const float* factor;
    int64_t sb, sh, ss;
    float scale;
    uint32_t H, n8;      // heads; eighths of the element count
};
struct CastJobs {
    CastJob job[3];
    uint32_t S;
};
int launch_cast_grads(const CastJobs& jobs, int count, bool fp16, cudaStream_t st);
// delta; `zero`, `zero_bytes`: 16-byte aligned memory to clear on the way (a multiple of 16 bytes), or null and 0.
int launch_delta(const void* out, const fmsa_tensor* d_out, float* delta, int B, int S, int Hq, int dtype, void* zero, int64_t zero_bytes,
                 cudaStream_t st);
int launch_sink_grad(const float* lse, const float* delta, const float* sinks, float* dsinks, int B, int S, int Hq, cudaStream_t st);

// What a whole pass has the reverse index do on the way.
struct RixWorkspace {       // scratch of the reverse index
    uint8_t* counts;        // [rows_bh][NB][NB] edges of (query tile, key block)
    int32_t* blk_off;       // [rows_bh][NB][NB] their offsets inside the reverse-index row
    int32_t* totals;        // [rows_bh][NB]
    size_t bytes;
};
RixWorkspace carve_reverse_index(void* base, int64_t rows_bh, int NB);
struct RixExtras {
    bool counted = false;           // the selection has filled `counts` and `visits` (select_fused_launch)
    void* visits = nullptr;         // [rows_bh][tiles][tiles] 128-bit words: which rows of query tile i selected block j
    int tiles = 0;
    int32_t* row_start = nullptr;   // [rows_bh*NB] position of the first row of a query tile >= tiles in every reverse-index row
    int32_t* zero = nullptr;        // words to clear
    int nzero = 0;
};
int reverse_index_launch(const int32_t* block_indices, int32_t* row_ptr, int32_t* col_q, int32_t* edge_pos, int64_t rows_bh,
                         int32_t S, int32_t Kb, void* scratch, cudaStream_t st, const RixExtras& x = RixExtras());
// The fused selection, and what the first step of the reverse index would read its result for: `counts` (see RixWorkspace) and
// x.visits, each where not null, and the words x.zero to clear.  `block_indices` null: only those.
int select_fused_launch(const fmsa_problem* pb, const fmsa_tensor* q_proxy, const fmsa_tensor* k_proxy, int32_t* block_indices,
                        uint8_t* counts, const RixExtras& x, int32_t* status, cudaStream_t st);
// Nothing but `visits` (and the cleared words).
int launch_tile_visits(const int32_t* block_indices, int64_t rows_bh, int32_t S, int32_t Kb, const RixExtras& x, cudaStream_t st);
int reverse_index_launches(int64_t rows_bh, int32_t S, const RixExtras& x);   // how many kernels that is
size_t reverse_index_scratch_bytes(int64_t rows_bh, int32_t S);

}  // namespace fmsa

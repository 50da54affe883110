// Whole passes in one call: the launch sequence of a forward and of a backward, with the division into (batch, KV head) group
// passes and the layout of the workspace.
//
// Why it is native: driven stage by stage from Python a training pass of B=1 S=1024 Hq=8 took 0.65 ms of host time against
// 0.11 ms of GPU time (a dozen ctypes calls, two dozen allocations, fills and copies of a few bytes).  One call, one workspace
// and no launch that only clears a word leave the autograd machinery as the larger part.
#include "host_common.h"
#include "launch.h"
#include "msa_common.cuh"

namespace fmsa {
namespace {

struct Carver {   // hands out 256-byte aligned pieces of one buffer
    char* base;
    int64_t off = 0;
    explicit Carver(void* p) : base(static_cast<char*>(p)) {}
    template <class T>
    T* take(int64_t count) {
        T* p = reinterpret_cast<T*>(base + off);
        off += round_up(count * static_cast<int64_t>(sizeof(T)), 256);
        return p;
    }
};

// Groups per pass, so that the partial rows of a pass stay within max_bytes (at least one group).
int64_t groups_per_pass(const fmsa_problem* pb, int dense, int64_t bytes_per_slot, int64_t max_bytes) {
    const int64_t groups = static_cast<int64_t>(pb->B) * pb->Hkv;
    const int64_t per = fmsa_fwd_partial_slots(pb, 1, dense) * bytes_per_slot;
    int64_t step = per > 0 ? max_bytes / per : groups;
    if (step < 1) step = 1;
    return step < groups ? step : groups;
}

struct ForwardSpace {
    int32_t* counters;    // one per pass of the key-block stationary forward, then the query-tile stationary one's
    int32_t* row_start;
    void* o_part;
    float* stats;
    int32_t* indices;
    float* scores;
    void *rix, *visits;
    int64_t gstep, slots, bytes;
    int tiles, passes;    // query tiles of the query-tile stationary forward; passes of the other one (0: all tiles are the former's)
};
// The selection's buffers and the partial rows of the key-block stationary forward, which comes last, are not alive at the same
// time: they share the space.
ForwardSpace carve_forward(const fmsa_problem* pb, int dense, int visible, int64_t max_bytes, void* base) {
    ForwardSpace w = {};
    w.tiles = forward_tiles(pb->S / kBlock, pb->top_k_blocks, static_cast<int64_t>(pb->B) * pb->Hq, dense, visible);
    const int mpp = pb->Hq / pb->Hp;
    const int64_t groups = static_cast<int64_t>(pb->B) * pb->Hkv, rows = static_cast<int64_t>(pb->B) * pb->Hp, NB = pb->S / 128;
    w.gstep = groups_per_pass(pb, dense, static_cast<int64_t>(mpp) * 256 + (mpp + 1) * 8, max_bytes);
    w.slots = fmsa_fwd_partial_slots(pb, static_cast<int32_t>(w.gstep), dense);
    w.passes = w.tiles < NB ? static_cast<int>((groups + w.gstep - 1) / w.gstep) : 0;
    Carver c(base);
    w.counters = c.take<int32_t>(w.passes + 1);
    if (w.passes) w.row_start = c.take<int32_t>(rows * NB);
    Carver a = c;
    if (w.passes) {
        w.o_part = a.take<uint16_t>(w.slots * mpp * 128);
        w.stats = a.take<float>(w.slots * (mpp + 1) * 2);
    }
    Carver s = c;
    if (!dense) {
        w.indices = s.take<int32_t>(rows * pb->S * pb->top_k_blocks);
        w.visits = s.take<char>(rows * w.tiles * w.tiles * 16);
        w.rix = s.take<char>(static_cast<int64_t>(reverse_index_scratch_bytes(rows, pb->S)));
        if (pb->top_k_blocks > FMSA_FUSED_SELECT_MAX_BLOCKS) w.scores = s.take<float>(rows * pb->S * NB);
    }
    w.bytes = a.off > s.off ? a.off : s.off;
    return w;
}

struct BackwardSpace {
    float *dk, *dv, *dkp;
    int32_t* counters;
    int64_t zero_bytes;   // dk, dv, dkp and the counters lie in front and are cleared by the delta kernel
    float* delta;
    void *dq_part, *dqp_part;
    int64_t gstep, slots, bytes;
    int split;
};
BackwardSpace carve_backward(const fmsa_problem* pb, int dense, int with_kl, int split_above, int64_t max_bytes, void* base) {
    BackwardSpace w = {};
    const int mpp = pb->Hq / pb->Hp;
    const int64_t groups = static_cast<int64_t>(pb->B) * pb->Hkv, tokens = static_cast<int64_t>(pb->B) * pb->S;
    const int edges = dense ? pb->S / 128 : pb->top_k_blocks;
    w.split = edges > split_above ? 1 : 0;
    const int planes = w.split ? 2 : 1;
    w.gstep = groups_per_pass(pb, dense, static_cast<int64_t>(mpp + (with_kl ? 1 : 0)) * 256 * planes, max_bytes);
    w.slots = fmsa_fwd_partial_slots(pb, static_cast<int32_t>(w.gstep), dense);
    Carver c(base);
    w.dk = c.take<float>(tokens * pb->Hkv * 128);
    w.dv = c.take<float>(tokens * pb->Hkv * 128);
    if (with_kl) w.dkp = c.take<float>(tokens * pb->Hpkv * 128);
    w.counters = c.take<int32_t>(2 * ((groups + w.gstep - 1) / w.gstep));
    w.zero_bytes = c.off;
    w.delta = c.take<float>(tokens * pb->Hq);
    w.dq_part = c.take<uint16_t>(planes * w.slots * mpp * 128);
    if (with_kl) w.dqp_part = c.take<uint16_t>(planes * w.slots * 128);
    w.bytes = c.off;
    return w;
}

// Optional timing marks around the stages.
struct Marks {
    fmsa_marks* m;
    cudaStream_t st;
    void operator()(int stage) {
        if (m && m->used < m->capacity) {
            m->stages[m->used] = stage;
            cudaEventRecord(static_cast<cudaEvent_t>(m->events[m->used++]), st);
        }
    }
};

}  // namespace
}  // namespace fmsa

#define FMSA_TRY(expr)                     \
    do {                                   \
        const int rc_ = (expr);            \
        if (rc_ != FMSA_OK) return rc_;    \
    } while (0)

extern "C" int64_t fmsa_forward_workspace_bytes(const fmsa_problem* pb, int32_t dense, int64_t max_partial_bytes) {
    return fmsa_forward_hinted_workspace_bytes(pb, dense, 0, max_partial_bytes);
}

extern "C" int64_t fmsa_forward_hinted_workspace_bytes(const fmsa_problem* pb, int32_t dense, int32_t visible, int64_t max_partial_bytes) {
    using namespace fmsa;
    return problem_ok(pb) ? carve_forward(pb, dense, visible, max_partial_bytes, nullptr).bytes : 0;
}

extern "C" int fmsa_forward(const fmsa_forward_args* a, fmsa_marks* marks, int32_t* launches, void* stream) {
    return fmsa_forward_hinted(a, 0, 0, marks, launches, stream);
}

extern "C" int fmsa_forward_hinted(const fmsa_forward_args* a, int32_t alone, int32_t visible, fmsa_marks* marks, int32_t* launches,
                                   void* stream) {
    using namespace fmsa;
    FMSA_REQUIRE(a && problem_ok(&a->pb) && a->workspace && a->out && a->lse && a->status && launches);
    FMSA_REQUIRE((reinterpret_cast<uintptr_t>(a->workspace) & 255u) == 0 && (!a->with_proxy || a->lse_proxy));
    const fmsa_problem* pb = &a->pb;
    const int dense = a->dense ? 1 : 0;
    FMSA_REQUIRE(dense || (pb->top_k_blocks >= 1 && pb->top_k_blocks <= pb->S / 128));
    const ForwardSpace w = carve_forward(pb, dense, visible, a->max_partial_bytes, a->workspace);
    const bool index = !dense && (!alone || w.passes);   // the reverse index is wanted
    FMSA_REQUIRE(!index || (a->row_ptr && a->col_q && a->edge_pos));
    if (w.bytes > a->workspace_bytes) return FMSA_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    Marks mark{marks, st};
    int n = 0;
    const int groups = pb->B * pb->Hkv, step = static_cast<int>(w.gstep);
    if (!dense) {
        const int64_t rows = static_cast<int64_t>(pb->B) * pb->Hp;
        FMSA_REQUIRE(rows <= 65535 && rows * pb->S * pb->top_k_blocks < 0x7fffffffLL);
        if (pb->S / 128 > 2048) return FMSA_ERR_UNSUPPORTED;
        // (the work counters and row_start lie outside the space that the selection's buffers share with the partial rows)
        RixExtras x;
        x.visits = w.visits; x.tiles = w.tiles; x.row_start = w.row_start;
        x.zero = w.counters; x.nzero = w.passes + 1;
        mark(FMSA_STAGE_SELECT);
        if (w.scores) {
            FMSA_TRY(fmsa_select_scores(&a->q_proxy, &a->k_proxy, w.scores, pb->B, pb->Hp, pb->Hpkv, pb->S, pb->scale, pb->dtype,
                                        pb->doc_start, a->status, stream));
            FMSA_TRY(fmsa_select_topk(w.scores, w.indices, rows, pb->S, pb->top_k_blocks, stream));
            n += 2;
        } else {
            x.counted = true;
            FMSA_TRY(select_fused_launch(pb, &a->q_proxy, &a->k_proxy, index ? w.indices : nullptr,
                                         index ? carve_reverse_index(w.rix, rows, pb->S / 128).counts : nullptr, x, a->status, st));
            n += 1;
        }
        mark(FMSA_STAGE_SELECT);
        mark(FMSA_STAGE_REVERSE_INDEX);
        if (index) {
            FMSA_TRY(reverse_index_launch(w.indices, a->row_ptr, a->col_q, a->edge_pos, rows, pb->S, pb->top_k_blocks, w.rix, st, x));
            n += reverse_index_launches(rows, pb->S, x);
        } else if (!x.counted) {
            FMSA_TRY(launch_tile_visits(w.indices, rows, pb->S, pb->top_k_blocks, x, st));
            n += 1;
        }
        mark(FMSA_STAGE_REVERSE_INDEX);
    } else if (cudaMemsetAsync(w.counters, 0, sizeof(int32_t) * (w.passes + 1), st) != cudaSuccess) {
        return FMSA_ERR_CUDA;
    }
    float* lse_proxy = a->with_proxy ? a->lse_proxy : nullptr;
    mark(FMSA_STAGE_ATTN_FWD);
    FMSA_TRY(launch_tile_fwd(pb, &a->q, &a->k, &a->v, &a->q_proxy, &a->k_proxy, w.visits, a->out, a->lse, lse_proxy, a->sinks, a->kl_loss,
                             w.tiles, dense, w.counters + w.passes, a->status, st));
    mark(FMSA_STAGE_ATTN_FWD);
    n += a->sinks ? 2 : 1;
    for (int i = 0; i < w.passes; ++i) {
        const int g0 = i * step, gc = groups - g0 < step ? groups - g0 : step;
        mark(FMSA_STAGE_ATTN_FWD);
        FMSA_TRY(launch_sparse_fwd(pb, &a->q, &a->k, &a->v, &a->q_proxy, &a->k_proxy, a->row_ptr, w.row_start, w.tiles, a->col_q, w.o_part,
                                   w.stats, w.slots, g0, gc, a->with_proxy, dense, w.counters + i, a->status, st));
        mark(FMSA_STAGE_ATTN_FWD);
        mark(FMSA_STAGE_FWD_COMBINE);
        FMSA_TRY(launch_fwd_combine(pb, w.o_part, w.stats, a->edge_pos, a->row_ptr, a->out, a->lse, lse_proxy, a->sinks, w.tiles, g0, gc, dense, st));
        mark(FMSA_STAGE_FWD_COMBINE);
        n += 3;
    }
    *launches = n;
    return FMSA_OK;
}

// ---------------------------------------------------------------------------------------------
// The query-tile stationary forward as a stage of its own.
// ---------------------------------------------------------------------------------------------
extern "C" int32_t fmsa_forward_tiles(const fmsa_problem* pb, int32_t dense, int32_t visible) {
    using namespace fmsa;
    return problem_ok(pb) ? forward_tiles(pb->S / kBlock, pb->top_k_blocks, static_cast<int64_t>(pb->B) * pb->Hq, dense, visible) : 0;
}

extern "C" int64_t fmsa_tile_fwd_workspace_bytes(const fmsa_problem* pb, int32_t dense) {
    using namespace fmsa;
    if (!problem_ok(pb)) return 0;
    const int64_t tiles = fmsa_forward_tiles(pb, dense, 0);
    return 256 + (dense ? 0 : static_cast<int64_t>(pb->B) * pb->Hp * tiles * tiles * 16);
}

extern "C" int fmsa_tile_fwd(const fmsa_problem* pb, const fmsa_tensor* q, const fmsa_tensor* k, const fmsa_tensor* v,
                             const fmsa_tensor* q_proxy, const fmsa_tensor* k_proxy, const int32_t* block_indices, void* workspace,
                             int64_t workspace_bytes, void* out, float* lse, float* lse_proxy, int32_t dense, int32_t* status,
                             void* stream) {
    using namespace fmsa;
    FMSA_REQUIRE(problem_ok(pb) && workspace && (reinterpret_cast<uintptr_t>(workspace) & 255u) == 0 && (dense || block_indices));
    FMSA_REQUIRE(dense || (pb->top_k_blocks >= 1 && pb->top_k_blocks <= pb->S / kBlock));
    if (workspace_bytes < fmsa_tile_fwd_workspace_bytes(pb, dense)) return FMSA_ERR_WORKSPACE;
    const int64_t rows = static_cast<int64_t>(pb->B) * pb->Hp;
    if (rows > 65535 || pb->S / kBlock > 2048) return FMSA_ERR_UNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RixExtras x;
    x.tiles = fmsa_forward_tiles(pb, dense, 0);
    x.zero = static_cast<int32_t*>(workspace); x.nzero = 1;
    if (!dense) {
        x.visits = static_cast<char*>(workspace) + 256;
        FMSA_TRY(launch_tile_visits(block_indices, rows, pb->S, pb->top_k_blocks, x, st));
    } else if (cudaMemsetAsync(workspace, 0, sizeof(int32_t), st) != cudaSuccess) {
        return FMSA_ERR_CUDA;
    }
    return launch_tile_fwd(pb, q, k, v, q_proxy, k_proxy, x.visits, out, lse, lse_proxy, nullptr, nullptr, x.tiles, dense, x.zero, status, st);
}

extern "C" int64_t fmsa_backward_workspace_bytes(const fmsa_problem* pb, int32_t dense, int32_t with_kl, int32_t split_above,
                                                 int64_t max_partial_bytes) {
    using namespace fmsa;
    return problem_ok(pb) ? carve_backward(pb, dense, with_kl, split_above, max_partial_bytes, nullptr).bytes : 0;
}

extern "C" int fmsa_backward(const fmsa_backward_args* a, fmsa_marks* marks, int32_t* launches, void* stream) {
    using namespace fmsa;
    FMSA_REQUIRE(a && problem_ok(&a->pb) && a->workspace && a->out && a->lse && a->status && launches);
    FMSA_REQUIRE(a->dq.ptr && a->dk.ptr && a->dv.ptr && a->dq_proxy.ptr && a->dk_proxy.ptr);
    FMSA_REQUIRE((reinterpret_cast<uintptr_t>(a->workspace) & 255u) == 0 && (!a->sinks || a->dsinks));
    const fmsa_problem* pb = &a->pb;
    const int dense = a->dense ? 1 : 0, kl = a->with_kl ? 1 : 0;
    const BackwardSpace w = carve_backward(pb, dense, kl, a->split_above, a->max_partial_bytes, a->workspace);
    if (w.bytes > a->workspace_bytes) return FMSA_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    Marks mark{marks, st};
    int n = 0;
    const int64_t tokens = static_cast<int64_t>(pb->B) * pb->S;
    FMSA_REQUIRE(tokens * (pb->Hkv > pb->Hpkv ? pb->Hkv : pb->Hpkv) * 16 < 0xffffffffLL);
    mark(FMSA_STAGE_DELTA);
    FMSA_TRY(launch_delta(a->out, &a->d_out, w.delta, pb->B, pb->S, pb->Hq, pb->dtype, a->workspace, w.zero_bytes, st));
    mark(FMSA_STAGE_DELTA);
    ++n;
    if (a->sinks) {
        FMSA_TRY(launch_sink_grad(a->lse, w.delta, a->sinks, a->dsinks, pb->B, pb->S, pb->Hq, st));
        ++n;
    }
    if (!kl) {   // (the views span their storage exactly: dense (B,H,S,128) or (B,S,H,128))
        if (cudaMemsetAsync(const_cast<void*>(a->dq_proxy.ptr), 0, static_cast<size_t>(tokens * pb->Hp * 256), st) != cudaSuccess ||
            cudaMemsetAsync(const_cast<void*>(a->dk_proxy.ptr), 0, static_cast<size_t>(tokens * pb->Hpkv * 256), st) != cudaSuccess)
            return FMSA_ERR_CUDA;
    }
    const int groups = pb->B * pb->Hkv, step = static_cast<int>(w.gstep), passes = (groups + step - 1) / step;
    for (int i = 0; i < passes; ++i) {
        const int g0 = i * step, gc = groups - g0 < step ? groups - g0 : step;
        mark(FMSA_STAGE_ATTN_BWD);
        FMSA_TRY(launch_sparse_bwd(pb, &a->q, &a->k, &a->v, &a->q_proxy, &a->k_proxy, &a->d_out, a->lse, kl ? a->lse_proxy : nullptr, w.delta,
                                   a->row_ptr, a->col_q, w.dq_part, w.dqp_part, w.slots, w.split, w.dkp, w.dk, w.dv, g0, gc, kl, dense,
                                   kl ? a->kl_value : nullptr, w.counters + 2 * i, w.counters + 2 * i + 1, false, a->status, st));
        mark(FMSA_STAGE_ATTN_BWD);
        mark(FMSA_STAGE_BWD_COMBINE);
        FMSA_TRY(fmsa_sparse_bwd_combine(pb, w.dq_part, w.dqp_part, w.slots, w.split, a->edge_pos, a->row_ptr, &a->dq,
                                         kl ? &a->dq_proxy : nullptr, a->grad_kl, g0, gc, dense, stream));
        mark(FMSA_STAGE_BWD_COMBINE);
        n += 2 + kl;
    }
    auto job = [&](const float* src, const fmsa_tensor& dst, int heads, float scale, const float* factor) {
        return CastJob{src, const_cast<void*>(dst.ptr), factor, dst.stride_b, dst.stride_h, dst.stride_s, scale, static_cast<uint32_t>(heads),
                       static_cast<uint32_t>(tokens * heads * 16)};
    };
    CastJobs jobs = {};
    jobs.S = static_cast<uint32_t>(pb->S);
    jobs.job[0] = job(w.dk, a->dk, pb->Hkv, pb->scale, nullptr);
    jobs.job[1] = job(w.dv, a->dv, pb->Hkv, 1.f, nullptr);
    if (kl) jobs.job[2] = job(w.dkp, a->dk_proxy, pb->Hpkv, pb->scale / (static_cast<float>(pb->B) * pb->Hp * pb->S), a->grad_kl);
    mark(FMSA_STAGE_CAST);
    FMSA_TRY(launch_cast_grads(jobs, 2 + kl, pb->dtype == FMSA_DTYPE_FP16, st));
    mark(FMSA_STAGE_CAST);
    *launches = n + 1;
    return FMSA_OK;
}

// ---------------------------------------------------------------------------------------------
// doc_start from document boundaries that the host holds: they travel as a kernel parameter, so that nothing is copied
// and nothing waits.
// ---------------------------------------------------------------------------------------------
namespace fmsa {
namespace {
struct DocBounds {
    int32_t n, per_batch;                       // boundaries per sequence; 1: a list per batch element, 0: one for all
    int32_t at[FMSA_MAX_HOST_BOUNDARIES];
};
__global__ void __launch_bounds__(256) doc_start_kernel(const __grid_constant__ DocBounds D, int32_t* __restrict__ doc_start, int S) {
    const int s = blockIdx.x * 256 + threadIdx.x, b = blockIdx.y;
    if (s >= S) return;
    const int32_t* at = D.at + (D.per_batch ? b * D.n : 0);
    int lo = 0, hi = D.n - 1;                   // last boundary <= s (boundary 0 is position 0, the last one is S)
    while (lo + 1 < hi) {
        const int mid = (lo + hi) >> 1;
        if (at[mid] <= s) lo = mid;
        else hi = mid;
    }
    doc_start[static_cast<int64_t>(b) * S + s] = at[lo];
}
}  // namespace
}  // namespace fmsa

extern "C" int fmsa_doc_start(const int32_t* boundaries, int32_t n, int32_t per_batch, int32_t B, int32_t S, int32_t* doc_start,
                              void* stream) {
    using namespace fmsa;
    FMSA_REQUIRE(boundaries && doc_start && n >= 2 && B > 0 && S > 0);
    const int64_t total = static_cast<int64_t>(n) * (per_batch ? B : 1);
    if (total > FMSA_MAX_HOST_BOUNDARIES || B > 65535) return FMSA_ERR_UNSUPPORTED;
    DocBounds D;
    D.n = n;
    D.per_batch = per_batch ? 1 : 0;
    for (int64_t i = 0; i < total; ++i) D.at[i] = boundaries[i];
    doc_start_kernel<<<dim3(static_cast<unsigned>((S + 255) / 256), static_cast<unsigned>(B)), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        D, doc_start, S);
    return check_launch();
}

// Proxy half of the fused MSA backward: dQp and dKp of the KL term, from the teacher that the main kernel
// (sparse_bwd.cu) left per edge.
//
// The same sub-units of the same reverse-index rows as in the main kernel; one tile per chunk of 128 gathered rows:
//     Sp^T  = Kp_j Qp_g^T                                      (both operands in shared memory; lane = key, column = query)
//     dSp^T = exp2(Sp^T*c - lse_proxy) - teacher/mpp           (fp32, rounded to 16 bit)
//     dQp   = dSp Kp_j                                         (dSp^T in shared memory)
//     dKp  += dSp^T Qp_g                                       (A operand in TMEM; accumulated over the sub-unit)
// (flash_msa/msa_backward_cutedsl.py:456-733, flash_msa/flash_msa.py:99-125.)  dQp leaves as 16-bit partial rows over the
// teacher it was formed from, dKp as fp32 reductions once per sub-unit.
//
// A tile reads 32 KB of teacher and 32 KB of gathered rows (mostly L2) and writes 32 KB: the memory rate bounds it (the three
// products are 1.5 k cycles of about 2.5 k).  So Sp^T of the next tile is issued ahead, the teacher words of the next tile are
// loaded into registers while this one is worked on, and three Qp stages keep the gathers ahead.
#include <cuda_fp16.h>

#include <type_traits>

#include "host_common.h"
#include "msa_common.cuh"
#include "proxy_bwd.h"
#include "sm100.cuh"
#include "tma_host.h"

namespace fmsa {
namespace {

struct ProxyParams {
    int32_t qp_row_b, qp_row_h, qp_row_s, qp_rows_total;   // row-gather view of q_proxy, as in the main kernel
    UnitSpace units;
    const int32_t* col_q;
    const int32_t* doc_start;
    const float* lse_proxy;    // [B,Hp,S]
    __nv_bfloat16* dqp_part;   // [slot][128]: teacher in, dQp out
    int64_t part_slots;        // slots per plane
    int split;                 // two planes (value, rounding remainder)
    float* dkp_acc;            // fp32 [B,Hpkv,S,128], zero-initialised
    int32_t* status;
    int S, Hp, Hpkv, pg;
    float scale_log2e, inv_mpp;
    float* kl_value;           // optional: += KL(teacher || proxy) summed over this launch's rows, / (B*Hp*S)
    float kl_value_scale;      // ln(2) / (B*Hp*S)
};

constexpr int kProxyUnitRing = 8, kProxyQStages = 3;
constexpr int kReads = 0, kDraws = 1, kOneThread = 2;   // how a role takes part in the common sequence of sub-units

struct alignas(16) ProxyRowStats {
    float neg_lse[128];    // -lse_proxy * log2(e); -inf for a dead row, whose probabilities then come out as 0
    uint8_t limit[128];    // last visible key of the row inside this key block (127 = all)
    uint8_t low[128];      // first visible key: document masking
};

struct ProxyCtrl {
    ProxyRowStats stats[2];
    uint64_t kp_full[2], kp_empty[2], acc_full, acc_free;
    uint64_t q_full[kProxyQStages], q_empty[kProxyQStages];
    uint64_t st_full[2], st_empty[2], s_full[2], ds_full[2], ds_free[2];
    uint64_t dq_full, dq_free;
    uint64_t unit_full[kProxyUnitRing];
    UnitRec units[kProxyUnitRing];
    int32_t any_low[2];
    uint32_t tmem_slot;
};

// Roles (warp index): 0-3, 4-7 compute (queries 0..63 and 64..127 of a tile), 8-11 output, 12-15 row gather, 16 Kp loads and
// row statistics, 17 MMA issue.  TMEM: Sp^T of even / odd tiles at columns 0 / 128 (dSp^T packed over it: queries 0..63 in
// columns 0..31, 64..127 in columns 64..95), dQp at 256 (lane = query), dKp at 384 (lane = key).
constexpr int kProxyThreads = 20 * 32;
constexpr int kProxyRegsCompute = 136, kProxyRegsOutput = 88, kProxyRegsGather = 56, kProxyRegsMisc = 64;
static_assert(2 * kProxyRegsCompute + kProxyRegsOutput + kProxyRegsGather + kProxyRegsMisc <= 5 * 96, "register re-division must balance");
constexpr size_t kProxyTileBytes = 7 * static_cast<size_t>(kTileBytes);   // Kp x2, Qp x3, dSp^T x2 (each also stages its dQp)
constexpr size_t kProxySmemBytes = 232448;
static_assert(kProxyTileBytes + sizeof(ProxyCtrl) <= kProxySmemBytes, "shared memory budget of one CTA");

template <bool FP16, bool VARLEN>
__global__ void __launch_bounds__(kProxyThreads, 1) proxy_bwd_kernel(const __grid_constant__ CUtensorMap tmap_qp,
                                                                     const __grid_constant__ CUtensorMap tmap_kp,
                                                                     const ProxyParams P) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t tiles = (smem_u32(smem_raw) + 1023u) & ~1023u;
    if ((tiles - smem_u32(smem_raw)) + kProxyTileBytes + sizeof(ProxyCtrl) > kProxySmemBytes) {
        wait_for_previous_kernel();   // (a kernel that has left counts as complete for those behind it)
        if (threadIdx.x == 0) atomicMax(P.status, kStatusBadSmem);
        return;
    }
    const uint32_t tile_kp0 = tiles, tile_q0 = tiles + 2 * kTileBytes, tile_ds0 = tiles + 5 * kTileBytes;
    ProxyCtrl* sm = reinterpret_cast<ProxyCtrl*>(smem_raw + (tiles - smem_u32(smem_raw)) + kProxyTileBytes);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;   // TMEM lane: key (compute, dKp read-out) or query (dQp read-out)
    auto BAR = [&](uint64_t& b) { return smem_u32(&b); };

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(BAR(sm->kp_full[i]), 1);
            mbar_init(BAR(sm->kp_empty[i]), 1);
            mbar_init(BAR(sm->st_full[i]), 1);
            mbar_init(BAR(sm->st_empty[i]), 8);
            mbar_init(BAR(sm->s_full[i]), 1);
            mbar_init(BAR(sm->ds_full[i]), 8);
            mbar_init(BAR(sm->ds_free[i]), 4);
        }
        for (int i = 0; i < kProxyQStages; ++i) {
            mbar_init(BAR(sm->q_full[i]), 4);
            mbar_init(BAR(sm->q_empty[i]), 1);
        }
        mbar_init(BAR(sm->dq_full), 1);
        mbar_init(BAR(sm->dq_free), 4);
        mbar_init(BAR(sm->acc_full), 1);
        mbar_init(BAR(sm->acc_free), 4);
        for (int i = 0; i < kProxyUnitRing; ++i) mbar_init(BAR(sm->unit_full[i]), 1);
        fence_mbar_init();
        prefetch_tmap(&tmap_qp);
        prefetch_tmap(&tmap_kp);
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(&sm->tmem_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    constexpr uint32_t tmem = 0, tmem_dq = 256, tmem_dkp = 384;   // all 512 columns: the allocation starts at column 0
    if (sm->tmem_slot != tmem) {
        wait_for_previous_kernel();   // (a kernel that has left counts as complete for those behind it)
        if (tid == 0) atomicMax(P.status, kStatusBadSmem);
        __syncthreads();
        if (warp == 0) tmem_dealloc(sm->tmem_slot, 512);
        return;
    }

    wait_for_previous_kernel();
    const int64_t edge_base = first_slot(P.units);
    bool bad = false;   // a bounded wait gave up (here or in another role): the thread stops taking work
    auto wait = [&](uint32_t bar, uint32_t parity) {   // every lane of the warp calls it; the result is warp-uniform
        if (!bad) bad = __any_sync(0xffffffffu, !mbar_wait_role(bar, parity));
    };
    auto wait1 = [&](uint32_t bar, uint32_t parity) {   // the same in a role that a single thread runs
        if (!bad) bad = !mbar_wait_role(bar, parity);
    };
    auto warp_arrive = [&](uint32_t bar) {
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
    };
    uint32_t gt = 0;     // tiles seen so far by this CTA (every role counts the same sequence)
    uint32_t nsub = 0;   // sub-units seen so far
    uint32_t qs = 0, qph = 0;   // gather warps / MMA issue: Qp stage of tile gt and the phase bit of its barriers
    float kl_acc = 0.f;
    auto next_unit = [&](uint32_t draw, UnitRec& ud, auto mode) -> bool {   // as in the main kernel
        const uint32_t uslot = draw & (kProxyUnitRing - 1);
        if (decltype(mode)::value == kDraws && warp == 12) {
            const UnitRec nu = draw_subunit(P.units);
            if (lane == 0) {
                sm->units[uslot] = nu;
                mbar_arrive(BAR(sm->unit_full[uslot]));
            }
        }
        if (decltype(mode)::value == kOneThread) wait1(BAR(sm->unit_full[uslot]), (draw / kProxyUnitRing) & 1);
        else wait(BAR(sm->unit_full[uslot]), (draw / kProxyUnitRing) & 1);
        if (bad) return false;
        ud = sm->units[uslot];
        return ud.chunk1 >= 0;
    };
    auto row_qid = [&](const UnitRec& ud, int at) -> int {
        if (at >= ud.n) return -1;
        const int q = P.units.dense ? (ud.j * kBlock + at) : P.col_q[ud.e0 + at];
        if (static_cast<unsigned>(q) >= static_cast<unsigned>(P.S) || (q >> 7) < ud.j) {
            atomicMax(P.status, kStatusBadIndex);
            return -1;
        }
        return q;
    };

    if (warp >= 16) {
        reg_dec<kProxyRegsMisc>();
        if (warp == 17 && elect_one()) {
            // =========================== MMA issue ===========================
            UnitRec ud;
            for (uint32_t draw = 0; next_unit(draw, ud, std::integral_constant<int, kOneThread>{}); ++draw, ++nsub) {
                const int ntiles = ud.chunk1 - ud.chunk0;
                const uint32_t kp = tile_kp0 + (nsub & 1) * kTileBytes;
                wait1(BAR(sm->kp_full[nsub & 1]), (nsub >> 1) & 1);
                uint32_t fs = qs, fph = qph;   // stage of the next Sp^T to issue
#pragma unroll 1
                for (int t = -1; t < ntiles && !bad; ++t) {
                    if (t + 1 < ntiles) {   // Sp^T runs one tile ahead
                        const uint32_t g = gt + (t >= 0 ? 1 : 0);
                        wait1(BAR(sm->q_full[fs]), fph);
                        // dKp of tile g - 2 (its Qp stage is the one after this) reads dSp^T from the columns that Sp^T overwrites:
                        // it must have completed, because products are only sure to follow one another where accumulator and
                        // shape are the same.
                        if (g >= 2) wait1(BAR(sm->q_empty[fs == kProxyQStages - 1 ? 0 : fs + 1]), ((g - 2) / kProxyQStages) & 1);
                        if (bad) break;
                        tc_fence_after_sync();
                        umma_tile_128<false, false, FP16>(tmem + (g & 1) * 128, kp, tile_q0 + fs * kTileBytes, false);
                        umma_commit(BAR(sm->s_full[g & 1]));
                        if (++fs == kProxyQStages) {
                            fs = 0;
                            fph ^= 1;
                        }
                    }
                    if (t < 0) continue;
                    const uint32_t b = gt & 1, s = tmem + b * 128;
                    wait1(BAR(sm->ds_full[b]), (gt >> 1) & 1);
                    if (gt >= 1) wait1(BAR(sm->dq_free), (gt - 1) & 1);
                    if (t == 0 && nsub > 0) wait1(BAR(sm->acc_free), (nsub - 1) & 1);
                    if (bad) break;
                    tc_fence_after_sync();
                    umma_tile_128<true, true, FP16>(tmem_dq, tile_ds0 + b * kTileBytes, kp, false);   // dQp = dSp Kp_j
                    umma_commit(BAR(sm->dq_full));
                    const uint32_t tq = tile_q0 + qs * kTileBytes;
                    umma_ts<4, 8, FP16>(tmem_dkp, s, tq, t != 0);                                   // dKp += dSp^T Qp_g
                    umma_ts<4, 8, FP16>(tmem_dkp, s + 64, tq + 64 * 128, true);
                    umma_commit(BAR(sm->q_empty[qs]));
                    if (++qs == kProxyQStages) {
                        qs = 0;
                        qph ^= 1;
                    }
                    ++gt;
                }
                if (!bad) {
                    umma_commit(BAR(sm->kp_empty[nsub & 1]));
                    umma_commit(BAR(sm->acc_full));
                }
            }
        } else if (warp == 16) {
            // =========================== Kp loads, row statistics ===========================
            UnitRec ud;
            for (uint32_t draw = 0; next_unit(draw, ud, std::integral_constant<int, kReads>{}); ++draw, ++nsub) {
                const uint32_t ks = nsub & 1;
                if (nsub >= 2) wait(BAR(sm->kp_empty[ks]), ((nsub >> 1) - 1) & 1);
                if (!bad && elect_one()) {
                    mbar_arrive_expect_tx(BAR(sm->kp_full[ks]), kTileBytes);
                    tma_load_tile(tile_kp0 + ks * kTileBytes, &tmap_kp, ud.j * kBlock, ud.p / P.pg, ud.b, BAR(sm->kp_full[ks]));
                }
                __syncwarp();
                const float* lse = P.lse_proxy + (static_cast<int64_t>(ud.b) * P.Hp + ud.p) * P.S;
                // Two dependent loads per row take longer than half a tile: positions are fetched two chunks ahead, the log-sum-exps one.
                int qid[4], next[4];
                float nl[4];
                auto fetch_positions = [&](int chunk) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) next[i] = chunk < ud.chunk1 ? row_qid(ud, chunk * kBlock + 4 * lane + i) : -1;
                };
                auto advance = [&](int chunk) {   // to chunk `chunk`
#pragma unroll
                    for (int i = 0; i < 4; ++i) qid[i] = next[i];
                    fetch_positions(chunk + 1);
#pragma unroll
                    for (int i = 0; i < 4; ++i) nl[i] = qid[i] >= 0 ? lse[qid[i]] : INFINITY;
                };
                fetch_positions(ud.chunk0);
                advance(ud.chunk0);
#pragma unroll 1
                for (int chunk = ud.chunk0; chunk < ud.chunk1; ++chunk, ++gt) {
                    const uint32_t s = gt & 1;
                    const float4 nl4 = make_float4(-kLog2e * nl[0], -kLog2e * nl[1], -kLog2e * nl[2], -kLog2e * nl[3]);
                    uint32_t lim4 = 0, low4 = 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int q = qid[i];
                        lim4 |= ((q >= 0 && (q >> 7) == ud.j) ? static_cast<uint32_t>(q & 127) : 127u) << (8 * i);
                        if (VARLEN && q >= 0) {
                            const int lo = P.doc_start[static_cast<int64_t>(ud.b) * P.S + q], lb = lo >> 7;
                            low4 |= static_cast<uint32_t>(lb < ud.j ? 0 : (lb == ud.j ? (lo & 127) : 128)) << (8 * i);
                        }
                    }
                    const bool any_low = VARLEN && __any_sync(0xffffffffu, low4 != 0);
                    advance(chunk + 1);
                    if (gt >= 2) wait(BAR(sm->st_empty[s]), ((gt >> 1) - 1) & 1);
                    if (bad) break;
                    ProxyRowStats* st = &sm->stats[s];
                    reinterpret_cast<float4*>(st->neg_lse)[lane] = nl4;
                    reinterpret_cast<uint32_t*>(st->limit)[lane] = lim4;
                    if (VARLEN) {
                        reinterpret_cast<uint32_t*>(st->low)[lane] = low4;
                        if (lane == 0) sm->any_low[s] = any_low ? 1 : 0;
                    }
                    warp_arrive(BAR(sm->st_full[s]));
                }
            }
        }
    } else if (warp >= 12) {
        reg_dec<kProxyRegsGather>();
        // =========================== row gather ===========================
        // Gather warp g fetches rows 32g .. 32g+31 of a tile: lanes 0..15 one gather4 each (row quad lane/2, 64-column panel lane%2).
        const int g = warp - 12;
        const int quad = (lane >> 1) & 7, panel = lane & 1;
        UnitRec ud;
        for (uint32_t draw = 0; next_unit(draw, ud, std::integral_constant<int, kDraws>{}); ++draw, ++nsub) {
            const int base = ud.b * P.qp_row_b + ud.p * P.qp_row_h;
            int next = row_qid(ud, ud.chunk0 * kBlock + 32 * g + lane);
#pragma unroll 1
            for (int chunk = ud.chunk0; chunk < ud.chunk1; ++chunk, ++gt) {
                const int q = next;
                if (chunk + 1 < ud.chunk1) next = row_qid(ud, (chunk + 1) * kBlock + 32 * g + lane);
                int r[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int qi = __shfl_sync(0xffffffffu, q, 4 * quad + i);
                    r[i] = qi >= 0 ? base + qi * P.qp_row_s : P.qp_rows_total;
                }
                if (gt >= kProxyQStages) wait(BAR(sm->q_empty[qs]), qph ^ 1);
                if (bad) break;
                const uint32_t full = BAR(sm->q_full[qs]);
                if (elect_one()) mbar_arrive_expect_tx(full, kTileBytes / 4);
                __syncwarp();
                if (lane < 16)
                    tma_gather4(tile_q0 + qs * kTileBytes + panel * kPanelBytes + (32 * g + 4 * quad) * 128, &tmap_qp, panel * 64, r[0], r[1], r[2], r[3], full);
                if (++qs == kProxyQStages) {
                    qs = 0;
                    qph ^= 1;
                }
            }
        }
    } else if (warp >= 8) {
        reg_dec<kProxyRegsOutput>();
        // =========================== output group ===========================
        UnitRec ud;
        for (uint32_t draw = 0; next_unit(draw, ud, std::integral_constant<int, kReads>{}); ++draw, ++nsub) {
            const int64_t slot_base = ud.e0 - edge_base;
#pragma unroll 1
            for (int chunk = ud.chunk0; chunk < ud.chunk1; ++chunk, ++gt) {
                wait(BAR(sm->dq_full), gt & 1);
                if (bad) break;
                tc_fence_after_sync();
                // Thread = row.  A warp stages its 32 rows in the tile's dSp^T (whose product is done), 64 columns at a time, and
                // stores them itself, 128 contiguous bytes of four rows per instruction: the four warps meet nowhere.  With two planes
                // the rounding remainders lie in the other panel.
                const uint32_t rows = tile_ds0 + (gt & 1) * kTileBytes + quarter * 32 * 128;
                const int r0 = lane >> 3;   // the lane stores rows r0 + 4 i of the warp's
                const int nrows = ud.n - chunk * kBlock - 32 * quarter - r0;
                __nv_bfloat16* to = P.dqp_part + (slot_base + static_cast<int64_t>(chunk) * kBlock + 32 * quarter + r0) * kHeadDim + 8 * (lane & 7);
#pragma unroll 1
                for (int c = 0; c < 128; c += 32) {
                    uint32_t v[32], pk[16];
                    tmem_ld32(tmem_addr(tmem_dq, quarter, c), v);
                    tmem_ld_wait();
                    if (c == 96) {
                        tc_fence_before_sync();
                        warp_arrive(BAR(sm->dq_free));
                    }
#pragma unroll
                    for (int i = 0; i < 16; ++i) pk[i] = pack_act<FP16>(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
                    uint32_t panel = rows + (P.split ? 0 : c >> 6) * kPanelBytes;
                    const int k0 = (c >> 3) & 4;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        st_shared_v4(panel + lane * 128 + (((k0 + k) ^ (lane & 7)) << 4), pk[4 * k], pk[4 * k + 1], pk[4 * k + 2], pk[4 * k + 3]);
                    if (P.split) {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            pk[i] = pack_act<FP16>(__uint_as_float(v[2 * i]) - act_lo<FP16>(pk[i]), __uint_as_float(v[2 * i + 1]) - act_hi<FP16>(pk[i]));
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            st_shared_v4(panel + kPanelBytes + lane * 128 + (((k0 + k) ^ (lane & 7)) << 4), pk[4 * k], pk[4 * k + 1], pk[4 * k + 2],
                                         pk[4 * k + 3]);
                    }
                    if (k0 == 0) continue;
                    __syncwarp();
                    __nv_bfloat16* dst = to + (c & 64);
#pragma unroll 1
                    for (int part = 0; part <= P.split; ++part) {
                        uint4 w[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) w[i] = ld_shared_v4(panel + (r0 + 4 * i) * 128 + (((lane ^ (r0 + 4 * i)) & 7) << 4));
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (4 * i < nrows) *reinterpret_cast<uint4*>(dst + 4 * i * kHeadDim) = w[i];
                        panel += kPanelBytes;
                        dst += P.part_slots * kHeadDim;
                    }
                    __syncwarp();   // the staging rows have been read
                }
                warp_arrive(BAR(sm->ds_free[gt & 1]));
            }
            if (bad) break;
            // dKp of the sub-unit: lane = key row of the block
            wait(BAR(sm->acc_full), nsub & 1);
            if (!bad) {
                tc_fence_after_sync();
                float* drow = P.dkp_acc + ((static_cast<int64_t>(ud.b) * P.Hpkv + ud.p / P.pg) * P.S + ud.j * kBlock + row) * kHeadDim;
#pragma unroll 1
                for (int c = 0; c < 128; c += 32) {
                    uint32_t v[32];
                    tmem_ld32(tmem_addr(tmem_dkp, quarter, c), v);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        red_add_v4(drow + c + i, __uint_as_float(v[i]), __uint_as_float(v[i + 1]), __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
                }
                tc_fence_before_sync();
                warp_arrive(BAR(sm->acc_free));
            }
        }
    } else {
        reg_inc<kProxyRegsCompute>();
        // =========================== compute groups ===========================
        // Thread = (key `row`, 64 queries of the tile).
        const int q0 = (warp >> 2) * 64;
        const float2 sc2 = make_float2(P.scale_log2e, P.scale_log2e);
        const float2 nim = make_float2(-P.inv_mpp, -P.inv_mpp);
        // teacher words of this thread's queries in chunk `chunk`; 0 beyond the end of the row
        auto load_teacher = [&](const UnitRec& ud, int chunk, uint32_t (&w)[32]) __attribute__((always_inline)) {
            const int64_t slot = ud.e0 - edge_base + static_cast<int64_t>(chunk) * kBlock + q0;
            int left = ud.n - chunk * kBlock - q0;
            const uint32_t* src = reinterpret_cast<const uint32_t*>(P.dqp_part) + slot * 64;
            if (left >= 64) {
#pragma unroll
                for (int g8 = 0; g8 < 8; ++g8) {
                    const uint4 v = *reinterpret_cast<const uint4*>(src + g8 * 512 + 4 * row);
                    w[4 * g8] = v.x; w[4 * g8 + 1] = v.y; w[4 * g8 + 2] = v.z; w[4 * g8 + 3] = v.w;
                }
                return;
            }
#pragma unroll 1
            for (int g8 = 0; g8 < 8; ++g8, left -= 8, src += 512) {
#pragma unroll
                for (int i = 0; i < 28; ++i) w[i] = w[i + 4];
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (left >= 8) {
                    v = *reinterpret_cast<const uint4*>(src + 4 * row);
                } else {
                    auto pair = [&](int i) -> uint32_t {
                        return 2 * i + 1 < left ? src[i * 128 + row] : 2 * i < left ? reinterpret_cast<const uint16_t*>(src + i * 128)[row] : 0u;
                    };
                    v = make_uint4(pair(0), pair(1), pair(2), pair(3));
                }
                w[28] = v.x; w[29] = v.y; w[30] = v.z; w[31] = v.w;
            }
        };
        uint32_t cur[32], nxt[32];
        UnitRec ud;
        for (uint32_t draw = 0; next_unit(draw, ud, std::integral_constant<int, kReads>{}); ++draw, ++nsub) {
            load_teacher(ud, ud.chunk0, cur);
#pragma unroll 1
            for (int chunk = ud.chunk0; chunk < ud.chunk1; ++chunk, ++gt) {
                if (chunk + 1 < ud.chunk1) load_teacher(ud, chunk + 1, nxt);
                const uint32_t b = gt & 1, ph = (gt >> 1) & 1;
                const uint32_t sc = tmem + b * 128 + q0;
                const uint32_t ds_row = tile_ds0 + b * kTileBytes + (warp >> 2) * kPanelBytes + row * 128;
                wait(BAR(sm->st_full[b]), ph);
                wait(BAR(sm->s_full[b]), ph);
                if (gt >= 2) wait(BAR(sm->ds_free[b]), ph ^ 1);   // the dQp of tile gt - 2 has left the tile
                if (bad) break;
                tc_fence_after_sync();
                const ProxyRowStats* st = &sm->stats[b];
                const bool own = chunk == 0;   // only the first chunk of a reverse-index row can hold rows of the key block itself
                if (P.kl_value) {   // KL(teacher || proxy) = sum t (ln t - ln p); t = 0 contributes nothing
#pragma unroll
                    for (int c = 0; c < 64; c += 16) {
                        uint32_t sv[16];
                        tmem_ld16(tmem_addr(sc, quarter, c), sv);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float2 tt = __half22float2(*reinterpret_cast<const __half2*>(&cur[(c + i) >> 1]));
                            const float tv = ((i & 1) ? tt.y : tt.x) * P.inv_mpp;
                            kl_acc += (tv > 0.f) ? tv * (fast_log2(tv) - (__uint_as_float(sv[i]) * P.scale_log2e + st->neg_lse[q0 + c + i])) : 0.f;
                        }
                    }
                }
                auto body = [&](auto masked_c) __attribute__((always_inline)) {
                    constexpr bool kMasked = decltype(masked_c)::value;
                    uint32_t sv[2][16];
                    tmem_ld16(tmem_addr(sc, quarter, 0), sv[0]);
#pragma unroll
                    for (int c = 0; c < 64; c += 16) {
                        const int cb = (c >> 4) & 1;
                        tmem_ld_wait();
                        if (c + 16 < 64) tmem_ld16(tmem_addr(sc, quarter, c + 16), sv[cb ^ 1]);
                        uint32_t dk[8];
#pragma unroll
                        for (int i4 = 0; i4 < 16; i4 += 4) {
                            const float4 nl4 = *reinterpret_cast<const float4*>(&st->neg_lse[q0 + c + i4]);
                            uint32_t lim = 0x7f7f7f7fu, lw = 0u;
                            if (kMasked) {
                                if (own) lim = *reinterpret_cast<const uint32_t*>(&st->limit[q0 + c + i4]);
                                if (VARLEN) lw = *reinterpret_cast<const uint32_t*>(&st->low[q0 + c + i4]);
                            }
#pragma unroll
                            for (int i2 = 0; i2 < 4; i2 += 2) {
                                const int i = i4 + i2;
                                const float2 nl2 = i2 ? make_float2(nl4.z, nl4.w) : make_float2(nl4.x, nl4.y);
                                const float2 a = f2_fma(f2_from_bits(sv[cb][i], sv[cb][i + 1]), sc2, nl2);   // log2 of the probability
                                float2 p = make_float2(fast_exp2(a.x), fast_exp2(a.y));
                                if (kMasked) {
                                    const int l0 = static_cast<int>((lim >> (8 * i2)) & 0xffu), l1 = static_cast<int>((lim >> (8 * i2 + 8)) & 0xffu);
                                    const int w0 = static_cast<int>((lw >> (8 * i2)) & 0xffu), w1 = static_cast<int>((lw >> (8 * i2 + 8)) & 0xffu);
                                    p.x = (row <= l0 && (!VARLEN || row >= w0)) ? p.x : 0.f;
                                    p.y = (row <= l1 && (!VARLEN || row >= w1)) ? p.y : 0.f;
                                }
                                const float2 d = f2_fma(__half22float2(*reinterpret_cast<const __half2*>(&cur[(c + i) >> 1])), nim, p);
                                dk[i >> 1] = pack_act<FP16>(d.x, d.y);
                            }
                        }
                        tmem_st8(tmem_addr(sc, quarter, c >> 1), dk);
                        st_shared_v4(ds_row + ((2 * c) ^ ((row & 7) << 4)), dk[0], dk[1], dk[2], dk[3]);
                        st_shared_v4(ds_row + ((2 * c + 16) ^ ((row & 7) << 4)), dk[4], dk[5], dk[6], dk[7]);
                    }
                };
                if (own || (VARLEN && sm->any_low[b] != 0)) body(std::true_type{});
                else body(std::false_type{});
                tmem_st_wait();
                fence_async_smem();
                tc_fence_before_sync();
                warp_arrive(BAR(sm->ds_full[b]));
                warp_arrive(BAR(sm->st_empty[b]));
#pragma unroll
                for (int i = 0; i < 32; ++i) cur[i] = nxt[i];
            }
        }
    }
    if (P.kl_value && warp < 8) {
        for (int o = 16; o > 0; o >>= 1) kl_acc += __shfl_xor_sync(0xffffffffu, kl_acc, o);
        if (lane == 0) atomicAdd(P.kl_value, kl_acc * P.kl_value_scale);
    }
    if (bad) {
        atomicMax(P.status, kStatusWaitTimeout);
        // Give loads and products that are still in flight time to finish before shared memory and TMEM are released.
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000) __nanosleep(1000);
    }
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace

int launch_proxy_bwd(const fmsa_problem* pb, const fmsa_tensor& q_proxy, const fmsa_tensor& k_proxy, const float* lse_proxy,
                     const UnitSpace& units, const int32_t* col_q, void* teacher_dqp, int64_t part_slots, int split,
                     float* dkp_acc, float* kl_value, int grid, int32_t* status, cudaStream_t stream) {
    const uint64_t qp_rows = gather_rows(pb->B, pb->Hp, pb->S, q_proxy.stride_b, q_proxy.stride_h, q_proxy.stride_s);
    CUtensorMap tqp, tkp;
    if (!make_tmap_gather(&tqp, q_proxy.ptr, qp_rows) ||
        !make_tmap_bhsd(&tkp, k_proxy.ptr, pb->B, pb->Hpkv, pb->S, k_proxy.stride_b, k_proxy.stride_h, k_proxy.stride_s, 128))
        return FMSA_ERR_CUDA;
    ProxyParams P;
    P.qp_row_b = static_cast<int32_t>(q_proxy.stride_b / 128); P.qp_row_h = static_cast<int32_t>(q_proxy.stride_h / 128);
    P.qp_row_s = static_cast<int32_t>(q_proxy.stride_s / 128); P.qp_rows_total = static_cast<int32_t>(qp_rows);
    P.units = units; P.col_q = col_q; P.doc_start = pb->doc_start; P.lse_proxy = lse_proxy;
    P.dqp_part = static_cast<__nv_bfloat16*>(teacher_dqp); P.part_slots = part_slots; P.split = split ? 1 : 0;
    P.dkp_acc = dkp_acc; P.status = status;
    P.S = pb->S; P.Hp = pb->Hp; P.Hpkv = pb->Hpkv; P.pg = pb->Hp / pb->Hpkv;
    P.scale_log2e = pb->scale * kLog2e; P.inv_mpp = static_cast<float>(pb->Hp) / static_cast<float>(pb->Hq);
    P.kl_value = kl_value;
    P.kl_value_scale = kLn2 / (static_cast<float>(pb->B) * pb->Hp * pb->S);
    using KernelFn = void (*)(CUtensorMap, CUtensorMap, ProxyParams);
    static const KernelFn kernels[4] = {proxy_bwd_kernel<false, false>, proxy_bwd_kernel<false, true>, proxy_bwd_kernel<true, false>,
                                        proxy_bwd_kernel<true, true>};
    const KernelFn kernel = kernels[(pb->dtype == FMSA_DTYPE_FP16 ? 2 : 0) + (pb->doc_start ? 1 : 0)];
    if (!ensure_smem_attr(reinterpret_cast<const void*>(kernel), kProxySmemBytes)) return FMSA_ERR_CUDA;
    launch_chained(kernel, grid, kProxyThreads, kProxySmemBytes, stream, tqp, tkp, P);
    return check_launch();
}

}  // namespace fmsa

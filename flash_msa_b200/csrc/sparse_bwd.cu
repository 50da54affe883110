// Fused MSA backward, key-block stationary: dQ, dK, dV and the on-the-fly KL gradients dQp, dKp.
//
// Work unit = (batch, KV head, key block j), exactly as in the forward: K_j and V_j stay in shared
// memory, the unit walks the reverse-index row of every proxy head of its group in chunks of 128
// gathered query rows.  For each chunk the main heads of the proxy head run one after another.  Scores
// are computed TRANSPOSED (TMEM lane = key, column = query) so that P^T and dS^T, written back into TMEM
// as 16-bit operands over the columns S^T occupied, are the TMEM operands of the dV and dK products:
//     S^T = K_j Q_g^T           dP^T = V_j dO_g^T                   (both operands in shared memory)
//     P^T = exp2(S^T*c - lse)   dS^T = P^T o (dP^T - delta)         (fp32, rounded to 16 bit)
//     dV += P^T dO_g            dK += dS^T Q_g                      (A operand in TMEM; accumulators stay in
//                                                                    TMEM for the whole sub-unit)
//     dQ^T = K_j^T dS^T                                             (dS^T also goes to shared memory)
// while every thread sums the P of its (key, queries) over the heads: the KL teacher, which is stored once per chunk.
// The proxy head's part runs as a kernel of its own behind this one (proxy_bwd.cu), from the teacher:
//     Sp^T = Kp_j Qp_g^T        p_px = exp2(Sp^T*c - lse_proxy)     dSp^T = p_px - teacher/mpp
//     dKp = dSp^T Qp_g, dQp = dSp Kp_j.
// As one more tile of every chunk it took twice the time of a main tile (its two halves need each other, its dKp does
// not fit TMEM beside dV and dK and left as 64 KB of fp32 reductions per chunk) and its code displaced the main tile's from
// the instruction cache.
// dQ and dQp leave as 16-bit per-edge partial rows (a combine kernel sums them per query row, applying
// scale and scale/(B*Hp*S)); dK and dV are added to fp32 accumulators with vector reductions once per sub-unit and
// cast afterwards.
//
// Formulas and rounding points follow the reference kernel
// (flash_msa/msa_backward_cutedsl.py:456-733: P and dS rounded to the input type before the
// second products, ds_px = c*(p_px - teacher)) and flash_msa/flash_msa.py:99-125 (delta, 1/(B*Hp*S),
// grad_kl applied afterwards on the device).  Differences: the teacher is summed from the unrounded P in
// fp16 pairs, and dSp is rounded to bf16 before the 1/(B*Hp*S) factor is applied.
// `dense` mode is the warmup backward (flash_msa/warmup/msa_backward_cutedsl_warmup.py:117-191):
// every causal (query block, key block) pair, with the schedule implied instead of built on the host.
#include <cuda_fp16.h>

#include <type_traits>

#include "host_common.h"
#include "launch.h"
#include "msa_common.cuh"
#include "proxy_bwd.h"
#include "sm100.cuh"
#include "tma_host.h"

namespace fmsa {
namespace {

#ifdef FMSA_TRACE
// Debug builds only: cycles each warp of CTA 0 spent inside its role (slot 0) and inside waits of kind 1..7.
__device__ unsigned long long g_bwd_trace[20][8];
#endif

struct BwdParams {
    // Row-gather views: element row (b, h, s) of q / d_out / q_proxy is matrix row b*row_b + h*row_h + s*row_s.
    int32_t q_row_b, q_row_h, q_row_s;
    int32_t do_row_b, do_row_h, do_row_s;
    int32_t q_rows_total, do_rows_total;   // first row index outside each view (reads as zeros)
    const float *lse, *delta;   // [B,Hq,S]
    UnitSpace units;
    const int32_t* col_q;
    const int32_t* doc_start;   // [B,S] first token of each token's document (packed sequences), or null
    __nv_bfloat16* dq_part;    // [(edge - edge_base) * mpp + head][128]: per-edge dQ contributions (unscaled)
    uint32_t* teacher;         // KL kernels: per edge 256 bytes (the dqp_part buffer), filled by the compute groups below
    int64_t part_slots;        // slots per plane of dq_part
    float *dk_acc, *dv_acc;    // fp32, zero-initialised, [B,Hkv,S,128]
    int32_t* status;
    int S, Hq, Hkv, mpp;
    float scale_log2e;
};

constexpr int kBwdUnitRing = 8;
constexpr int kReads = 0, kDraws = 1, kOneThread = 2;   // how a role takes part in the common sequence of sub-units

// Per-tile facts about the 128 gathered query rows (= TMEM columns), staged for the compute groups.
struct alignas(16) BwdRowStats {   // (filled and read with 16-byte vector accesses)
    float neg_lse[128];    // -lse * log2(e); -inf for a dead row, whose probabilities then come out as 0
    float neg_delta[128];  // -delta
    uint8_t limit[128];    // last visible key of the row inside this key block (127 = all)
    uint8_t low[128];      // first visible key (0 = all, 128 = none): document masking; written only with documents
};

struct BwdCtrl {
    uint64_t kv_full, kv_empty, acc_full, acc_free;
    uint64_t qdo_full[2][2], qdo_empty[2][2];    // [stage][half]
    uint64_t st_full[2], st_empty[2];
    uint64_t sdp_full[2], pds_full[2], dq_full[2], dq_free[2], ds_free[2];   // [half]
    uint64_t unit_full[kBwdUnitRing];
    UnitRec units[kBwdUnitRing];
    BwdRowStats stats[2];
    int32_t any_low[2];          // some row of the tile has low > 0 (document masking)
    uint32_t tmem_slot;
};

// Roles (warp index): 0-3 compute group A (queries 0..31 of a half tile), 4-7 compute group B (queries 32..63),
// 8-11 output group, 12-15 row gather (Q, dO), 16 K/V loads and row statistics, 17 MMA issue (18, 19 only
// take part in the block-wide steps).  A TMA row gather costs the issuing warp ~65 cycles whatever its size, so the
// 128 gathers of a tile are spread over four warps.
constexpr int kBwdGatherWarps = 4;
constexpr int kBwdThreads = 20 * 32;
// Registers per thread after the warpgroups re-divide the register file (setmaxnreg).  A CTA of 640 threads is
// launched with 96 registers per thread; an increase can only be served from what the other warpgroups of the
// same CTA gave up, so the five warpgroups must not ask for more than 5 x 96 in total (a warpgroup that asks for
// registers nobody released waits forever).
constexpr int kBwdRegsLaunch = 96, kBwdRegsCompute = 136, kBwdRegsOutput = 88, kBwdRegsGather = 56, kBwdRegsMisc = 64;
static_assert(2 * kBwdRegsCompute + kBwdRegsOutput + kBwdRegsGather + kBwdRegsMisc <= 5 * kBwdRegsLaunch,
              "register re-division must balance");
static_assert(kBwdRegsLaunch == (65536 / kBwdThreads) / 8 * 8, "registers per thread at launch");
constexpr size_t kBwdTileBytes = 7 * static_cast<size_t>(kTileBytes);   // K, V, Q x2, dO x2, dS^T
constexpr size_t kBwdSmemBytes = 232448;                                 // everything a CTA can have
static_assert(kBwdTileBytes + sizeof(BwdCtrl) <= kBwdSmemBytes, "shared memory budget of one CTA");
constexpr uint32_t kHalfRowBytes = 64 * 128;   // rows 64.. of a panel: where half 1 of a gathered tile starts

// Warp-specialised backward.  Every role walks the same sequence of sub-units (published by the gather warp in a
// ring) and of tiles.  A tile is worked on as two halves of 64 queries, x = 0 and 1, that take turns on the tensor core:
// while the compute groups turn S^T, dP^T of one half into P^T, dS^T, the products of the other half run.  TMEM (512 columns):
//   Rx [128x, 128x+128), x = 0, 1: columns 0..63 S^T of the half, overwritten in place by P^T and dS^T (16 bit; 16 queries
//                at a time: 8 columns of P^T, then 8 of dS^T); columns 64..127 dP^T, then dQ^T (lane = head dimension).
//   R2 [256,384) dV, R3 [384,512) dK (lane = key), accumulated over the sub-unit.
// A step of the issuing warp (half x of main tile t), behind P^T / dS^T of that half:
//   dQ^T = K^T dS^T -> Rx+64,  dV += P^T dO,  dK += dS^T Q,  [these complete]  S^T(t+1) = K Q^T -> Rx,  [dQ^T read out]
//   dP^T(t+1) = V dO^T -> Rx+64
// so dQ^T is read out under three products, and everything half x needs for tile t+1 is under way before the step of the
// other half begins.  (As one 128-query tile whose products, arithmetic and hand-offs followed one another, a tile took 8.1 k
// cycles, 4.0 k of them products: S^T, dP^T, dV and dK of 128 queries fill the 512 columns, and nothing of the next tile
// could start before dQ had been read out.)
// Hand-offs (mbarriers; one arrival per warp or per tcgen05.commit): qdo_full (TMA bytes) <- qdo_empty (dV, dK have read the
// rows, and the half's P^T, dS^T); st_full <- st_empty (row statistics); sdp_full (S^T and dP^T of a half), pds_full (P^T, dS^T written), dq_full -> dq_free (dQ^T read out),
// ds_free (the half's panel of the dS^T tile, which doubles as the staging tile of its dQ store, is reusable),
// acc_full / acc_free (dV, dK flushed at the end of a sub-unit).
// VARLEN: document masking of packed sequences (P.doc_start given).  A separate instantiation, so that the plain kernel
// carries none of its registers or code.  SPLIT: two planes of partial rows.
template <bool FP16, bool VARLEN, bool KL, bool SPLIT>
__global__ void __launch_bounds__(kBwdThreads, 1) sparse_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q,
                                                                    const __grid_constant__ CUtensorMap tmap_do,
                                                                    const __grid_constant__ CUtensorMap tmap_k,
                                                                    const __grid_constant__ CUtensorMap tmap_v,
                                                                    const BwdParams P) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t tiles = (smem_u32(smem_raw) + 1023u) & ~1023u;
    if ((tiles - smem_u32(smem_raw)) + kBwdTileBytes + sizeof(BwdCtrl) > kBwdSmemBytes) {
        wait_for_previous_kernel();   // (a kernel that has left counts as complete for those behind it)
        if (threadIdx.x == 0) atomicMax(P.status, kStatusBadSmem);
        return;
    }
    const uint32_t tile_k = tiles, tile_v = tiles + kTileBytes;
    const uint32_t tile_q0 = tiles + 2 * kTileBytes, tile_do0 = tiles + 4 * kTileBytes, tile_ds = tiles + 6 * kTileBytes;
    BwdCtrl* sm = reinterpret_cast<BwdCtrl*>(smem_raw + (tiles - smem_u32(smem_raw)) + kBwdTileBytes);

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;   // TMEM lane of this thread: key (compute, dV/dK read-out)
    auto BAR = [&](uint64_t& b) { return smem_u32(&b); };

    if (tid == 0) {
        mbar_init(BAR(sm->kv_full), 1);
        mbar_init(BAR(sm->kv_empty), 1);
        mbar_init(BAR(sm->acc_full), 1);
        mbar_init(BAR(sm->acc_free), 4);
        for (int i = 0; i < 2; ++i) {
            for (int x = 0; x < 2; ++x) {
                mbar_init(BAR(sm->qdo_full[i][x]), kBwdGatherWarps / 2);
                mbar_init(BAR(sm->qdo_empty[i][x]), 1);
            }
            mbar_init(BAR(sm->st_full[i]), 1);
            mbar_init(BAR(sm->st_empty[i]), 8);
            mbar_init(BAR(sm->sdp_full[i]), 1);
            mbar_init(BAR(sm->pds_full[i]), 8);
            mbar_init(BAR(sm->dq_full[i]), 1);
            mbar_init(BAR(sm->dq_free[i]), 4);
            mbar_init(BAR(sm->ds_free[i]), 4);
        }
        for (int i = 0; i < kBwdUnitRing; ++i) mbar_init(BAR(sm->unit_full[i]), 1);
        fence_mbar_init();
        prefetch_tmap(&tmap_q);
        prefetch_tmap(&tmap_do);
        prefetch_tmap(&tmap_k);
        prefetch_tmap(&tmap_v);
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(&sm->tmem_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    // All 512 columns are this CTA's, so the allocation starts at column 0 and every TMEM address is a constant.
    constexpr uint32_t tmem = 0;
    if (sm->tmem_slot != tmem) {
        wait_for_previous_kernel();   // (a kernel that has left counts as complete for those behind it)
        if (tid == 0) atomicMax(P.status, kStatusBadSmem);
        __syncthreads();
        if (warp == 0) tmem_dealloc(sm->tmem_slot, 512);
        return;
    }
    const uint32_t r2 = tmem + 256, r3 = tmem + 384;   // (Rx = tmem + 128 * x)

    const int hpc = P.mpp;   // tiles per chunk
    wait_for_previous_kernel();
    const int64_t edge_base = first_slot(P.units);
    bool bad = false;   // a bounded wait gave up (here or in another role): the thread stops taking work
#ifdef FMSA_TRACE
    unsigned long long trace_acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const long long trace_t0 = clock64();
#endif
    auto wait = [&](uint32_t bar, uint32_t parity, int kind = 1) {   // every lane of the warp calls it; the result is warp-uniform
#ifdef FMSA_TRACE
        const long long w0 = clock64();
#endif
        if (!bad) bad = __any_sync(0xffffffffu, !mbar_wait_role(bar, parity));
#ifdef FMSA_TRACE
        trace_acc[kind & 7] += static_cast<unsigned long long>(clock64() - w0);
#endif
        (void)kind;
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

    // Next sub-unit of the common sequence (false: no more work, or the CTA is giving up).  The gather warp draws the
    // work and publishes the decoded sub-unit; it passes over sub-units that lie beyond the end of their row, so
    // every published entry has work (or is the end marker).  The roles are at most a few tiles apart, fewer than the
    // ring has entries.
    auto next_unit = [&](uint32_t draw, UnitRec& ud, auto mode) -> bool {
        const uint32_t uslot = draw & (kBwdUnitRing - 1);
        if (decltype(mode)::value == kDraws && warp == 12) {
            const UnitRec nu = draw_subunit(P.units);
            if (lane == 0) {
                sm->units[uslot] = nu;
                mbar_arrive(BAR(sm->unit_full[uslot]));
            }
        }
        if (decltype(mode)::value == kOneThread) wait1(BAR(sm->unit_full[uslot]), (draw / kBwdUnitRing) & 1);
        else wait(BAR(sm->unit_full[uslot]), (draw / kBwdUnitRing) & 1, 7);
        if (bad) return false;
        ud = sm->units[uslot];
        return ud.chunk1 >= 0;
    };
    // query position of row `at` of a reverse-index row, -1 when there is none (or the index is bad)
    auto row_qid = [&](const UnitRec& ud, int at) -> int {
        if (at >= ud.n) return -1;
        const int q = P.units.dense ? (ud.j * kBlock + at) : P.col_q[ud.e0 + at];
        if (static_cast<unsigned>(q) >= static_cast<unsigned>(P.S) || (q >> 7) < ud.j) {
            atomicMax(P.status, kStatusBadIndex);
            return -1;
        }
        return q;
    };

    // Every role has its own loop over the common sequence of sub-units (separate loops keep the register
    // allocation of one role from being charged with the live values of the others).
    if (warp >= 16) {
        reg_dec<kBwdRegsMisc>();
        if (warp == 17 && elect_one()) {
            // =========================== MMA issue ===========================
            // One thread runs the whole role.  The tensor core holds a handful of instructions that have not started, i.e.
            // about 200 cycles of work: whatever the issuing thread does between two products in more than that is time the
            // tensor core stands still, so barriers are looked at before the product that precedes their use is issued.
            UnitRec ud;
            for (uint32_t draw = 0; next_unit(draw, ud, std::integral_constant<int, kOneThread>{}); ++draw, ++nsub) {
                const int ntiles = (ud.chunk1 - ud.chunk0) * hpc;
                wait1(BAR(sm->kv_full), nsub & 1);
                // One step per half tile: the products of (tile t, half x), then the front (S^T and dP^T) of that half of the next
                // tile; at the start (u = -1) the front of both halves.
                bool pds_ready = false;              // the next step's operands have been seen written
#pragma unroll 1
                for (int u = -1; u < 2 * ntiles && !bad; ++u) {
                    const int x = u & 1;
                    const uint32_t rx = tmem + 128 * x;
                    if (u >= 0) {
                        const uint32_t s = gt & 1;
                        const uint32_t tq = tile_q0 + s * kTileBytes + x * kHalfRowBytes, tdo = tile_do0 + s * kTileBytes + x * kHalfRowBytes;
                        if (!pds_ready) wait1(BAR(sm->pds_full[x]), gt & 1);
                        if (bad) break;
                        tc_fence_after_sync();
                        umma_ss<64, 8, true, true, FP16>(rx + 64, tile_k, tile_ds + x * kPanelBytes, false);   // dQ^T = K_j^T dS^T
                        umma_commit(BAR(sm->dq_full[x]));
                        if (u == 0 && nsub > 0) {
                            wait1(BAR(sm->acc_free), (nsub - 1) & 1);   // dV, dK of the previous sub-unit flushed
                            if (bad) break;
                            tc_fence_after_sync();
                        }
                        umma_ts<4, 16, FP16>(r2, rx, tdo, u != 0);       // dV += P^T dO_g
                        umma_ts<4, 16, FP16>(r3, rx + 8, tq, u != 0);    // dK += dS^T Q_g
                        umma_commit(BAR(sm->qdo_empty[s][x]));
                    }
                    pds_ready = false;
                    if (u + 2 < 2 * ntiles) {
                        const uint32_t g = u < 0 ? gt : gt + 1, s = g & 1;
#pragma unroll 1
                        for (int fx = u < 0 ? 0 : x; fx <= x; ++fx) {
                            const uint32_t rf = tmem + 128 * fx;
                            wait1(BAR(sm->qdo_full[s][fx]), (g >> 1) & 1);
                            // dV and dK of the half's previous tile read P^T, dS^T from the columns that S^T overwrites: they must
                            // have completed, because products are only sure to follow one another where accumulator and shape
                            // are the same.  (At B=2 S=8192 Hq=32 top-k 16 blocks the wait takes this kernel from 1.161 to
                            // 1.192 ms without KL work, the two backward kernels from 1.586 to 1.594 ms with it; dQ^T issued behind
                            // dV and dK, so that the tensor core has work meanwhile, 1.237 and 1.640: dQ^T is read out later.)
                            if (g >= 1) wait1(BAR(sm->qdo_empty[s ^ 1][fx]), ((g - 1) >> 1) & 1);
                            if (bad) break;
                            tc_fence_after_sync();
                            umma_ss<64, 8, false, false, FP16>(rf, tile_k, tile_q0 + s * kTileBytes + fx * kHalfRowBytes, false);   // S^T = K_j Q_g^T
                            if (u >= 0) pds_ready = mbar_try_wait(BAR(sm->pds_full[x ^ 1]), (gt + x) & 1);
                            if (g >= 1) {
                                wait1(BAR(sm->dq_free[fx]), (g - 1) & 1);   // dQ^T has been read out
                                if (bad) break;
                                tc_fence_after_sync();
                            }
                            umma_ss<64, 8, false, false, FP16>(rf + 64, tile_v, tile_do0 + s * kTileBytes + fx * kHalfRowBytes, false);   // dP^T = V_j dO_g^T
                            umma_commit(BAR(sm->sdp_full[fx]));
                        }
                    }
                    if (u >= 0 && x == 1) ++gt;
                }
                if (!bad) umma_commit(BAR(sm->kv_empty));
                if (!bad) umma_commit(BAR(sm->acc_full));
            }
        } else if (warp == 16) {
            // =========================== K / V loads, row statistics ===========================
            UnitRec ud;
            for (uint32_t draw = 0; next_unit(draw, ud, std::integral_constant<int, kReads>{}); ++draw, ++nsub) {
                if (nsub > 0) wait(BAR(sm->kv_empty), (nsub - 1) & 1, 1);
                if (!bad && elect_one()) {
                    mbar_arrive_expect_tx(BAR(sm->kv_full), 2 * kTileBytes);
#pragma unroll 1
                    for (int i = 0; i < 4; ++i)   // two panels of K_j, two of V_j
                        tma_load_4d(tile_k + i * kPanelBytes, i < 2 ? &tmap_k : &tmap_v, (i & 1) * 64, ud.j * kBlock, ud.kvh, ud.b, BAR(sm->kv_full));
                }
                __syncwarp();
                // per head: -lse * log2 e and -delta of the 128 rows
                const int64_t head0 = (static_cast<int64_t>(ud.b) * P.Hq + ud.p * P.mpp) * P.S;
#pragma unroll 1
                for (int chunk = ud.chunk0; chunk < ud.chunk1 && !bad; ++chunk) {
                    int qid[4];
                    uint32_t lim4 = 0, low4 = 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        qid[i] = row_qid(ud, chunk * kBlock + 4 * lane + i);
                        const uint32_t lim = (qid[i] >= 0 && (qid[i] >> 7) == ud.j) ? static_cast<uint32_t>(qid[i] & 127) : 127u;
                        lim4 |= lim << (8 * i);
                        if (VARLEN && qid[i] >= 0) {
                            const int lo = P.doc_start[static_cast<int64_t>(ud.b) * P.S + qid[i]];
                            const int lb = lo >> 7;
                            low4 |= static_cast<uint32_t>(lb < ud.j ? 0 : (lb == ud.j ? (lo & 127) : 128)) << (8 * i);
                        }
                    }
                    const bool any_low = VARLEN && __any_sync(0xffffffffu, low4 != 0);
                    const float *lse_row = P.lse + head0, *delta_row = P.delta + head0;
#pragma unroll 1
                    for (int hh = 0; hh < hpc; ++hh, ++gt) {
                        const uint32_t s = gt & 1;
                        float nl[4], dl[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            nl[i] = qid[i] >= 0 ? -kLog2e * lse_row[qid[i]] : -INFINITY;
                            dl[i] = qid[i] >= 0 ? -delta_row[qid[i]] : 0.f;
                        }
                        lse_row += P.S;
                        delta_row += P.S;
                        if (gt >= 2) wait(BAR(sm->st_empty[s]), ((gt >> 1) - 1) & 1, 2);
                        if (bad) break;
                        BwdRowStats* st = &sm->stats[s];
                        reinterpret_cast<float4*>(st->neg_lse)[lane] = make_float4(nl[0], nl[1], nl[2], nl[3]);
                        reinterpret_cast<float4*>(st->neg_delta)[lane] = make_float4(dl[0], dl[1], dl[2], dl[3]);
                        reinterpret_cast<uint32_t*>(st->limit)[lane] = lim4;
                        if (VARLEN) {
                            reinterpret_cast<uint32_t*>(st->low)[lane] = low4;
                            if (lane == 0) sm->any_low[s] = any_low ? 1 : 0;
                        }
                        warp_arrive(BAR(sm->st_full[s]));
                    }
                }
            }
        }
    } else if (warp >= 12) {
        reg_dec<kBwdRegsGather>();
        // =========================== row gather ===========================
        // Gather warp g fetches rows 32g .. 32g+31 of every tile, i.e. warps 0, 1 half 0 and warps 2, 3 half 1: lanes 0..15
        // issue the dO rows, lanes 16..31 the Q rows; a lane takes row quad (lane/2)%8 and 64-column panel lane%2.  Lane r
        // holds the query position of row 32g + r.
        const int g = warp - 12, half = g >> 1;
        const int quad = (lane >> 1) & 7, panel = lane & 1;
        const bool q_lane = lane >= 16;
        const int main_row_h = q_lane ? P.q_row_h : P.do_row_h, main_row_s = q_lane ? P.q_row_s : P.do_row_s;
        const int main_rows_total = q_lane ? P.q_rows_total : P.do_rows_total;
        const void* main_tmap = q_lane ? static_cast<const void*>(&tmap_q) : static_cast<const void*>(&tmap_do);
        UnitRec ud;
        for (uint32_t draw = 0; next_unit(draw, ud, std::integral_constant<int, kDraws>{}); ++draw, ++nsub) {
            // matrix row of (this lane's tensor, first main head, position 0); row numbers fit 31 bits
            const int main_base = q_lane ? ud.b * P.q_row_b + ud.p * P.mpp * P.q_row_h : ud.b * P.do_row_b + ud.p * P.mpp * P.do_row_h;
            for (int chunk = ud.chunk0; chunk < ud.chunk1 && !bad; ++chunk) {
                const int q = row_qid(ud, chunk * kBlock + 32 * g + lane);
                int qr[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) qr[i] = __shfl_sync(0xffffffffu, q, 4 * quad + i);
                for (int hh = 0; hh < hpc && !bad; ++hh, ++gt) {
                    const uint32_t s = gt & 1, ph = (gt >> 1) & 1;
                    const uint32_t full = BAR(sm->qdo_full[s][half]);
                    const uint32_t off = panel * kPanelBytes + (32 * g + 4 * quad) * 128;
                    if (gt >= 2) wait(BAR(sm->qdo_empty[s][half]), ph ^ 1, 1);
                    if (bad) break;
                    if (elect_one()) mbar_arrive_expect_tx(full, 2 * kTileBytes / kBwdGatherWarps);   // this warp's rows of both tiles
                    __syncwarp();
                    // One issue site for both tensors: every lane's gather4 goes through the uniform registers by itself, so each
                    // site is a loop of its own in the code.
                    const int base = main_base + hh * main_row_h;
                    int r[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) r[i] = qr[i] >= 0 ? base + qr[i] * main_row_s : main_rows_total;
                    const uint32_t dst = (q_lane ? tile_q0 : tile_do0) + s * kTileBytes + off;
                    tma_gather4(dst, main_tmap, panel * 64, r[0], r[1], r[2], r[3], full);
                }
            }
        }
    } else if (warp >= 8) {
        reg_dec<kBwdRegsOutput>();
        // =========================== output group ===========================
        UnitRec ud;
        for (uint32_t draw = 0; next_unit(draw, ud, std::integral_constant<int, kReads>{}); ++draw, ++nsub) {
            const int ntiles = (ud.chunk1 - ud.chunk0) * hpc;
            const int64_t slot_base = ud.e0 - edge_base;
            int hh = 0, chunk = ud.chunk0;
            for (int t = 0; t < ntiles && !bad; ++t, ++gt) {
                const int64_t slot0 = slot_base + static_cast<int64_t>(chunk) * kBlock;
#pragma unroll 1
                for (int x = 0; x < 2; ++x) {
                    wait(BAR(sm->dq_full[x]), gt & 1, 2);
                    if (bad) break;
                    tc_fence_after_sync();
                    // dQ^T (lane = head dimension, column = query of the half) -> 16 bit -> transposed into the half's panel of
                    // the dS^T tile (its products are done), from where it leaves as rows of one query.  Every warp stages and
                    // stores its own 32 head dimensions, 64 bytes of a row, so that the four warps meet nowhere (storing whole rows
                    // of 256 bytes took two barriers per store, during which the panel was held: 1.17 -> 1.14 ms without KL work).
                    // With SPLIT the rows leave twice: rounded, and the remainder of that rounding (a second
                    // plane of the partial buffers, `part_slots` slots further on), so that the sum over many edges keeps
                    // fp32-like accuracy.
                    const uint32_t src = tmem + 128 * x + 64 + (static_cast<uint32_t>(quarter * 32) << 16);
                    const uint32_t stage = tile_ds + x * kPanelBytes + quarter * (kPanelBytes / 4);   // 64 rows of 64 bytes, swizzled
                    const int r0 = lane >> 2;                                                  // the lane stores rows r0 + 8 i
                    const int nrows = min(64, ud.n - chunk * kBlock - 64 * x) - r0;            // <= 0: nothing to write
                    __nv_bfloat16* to = P.dq_part + ((slot0 + 64 * x + r0) * P.mpp + hh) * kHeadDim + 32 * quarter + 8 * (lane & 3);
                    const uint32_t from = stage + r0 * 64 + (((lane ^ (r0 >> 1)) & 3) << 4);
                    // stmatrix: lane l addresses row l%8 of block l/8; blocks are (queries +0, dims +0), (+0, +8), (+8, +0), (+8, +8)
                    const uint32_t into = stage + ((lane >> 4) * 8 + (lane & 7)) * 64;
                    const int64_t row8 = static_cast<int64_t>(8 * P.mpp) * kHeadDim;
                    if constexpr (!SPLIT) {
#pragma unroll 1
                        for (int i = 0; i < 2; ++i) {   // 16 head-dimension lanes of the warp's 32 at a time
                            uint32_t v[32], pk[16];
                            tmem_ld_16x256_x8(src + (static_cast<uint32_t>(16 * i) << 16), v);
                            tmem_ld_wait();
                            if (i == 1) {
                                tc_fence_before_sync();
                                warp_arrive(BAR(sm->dq_free[x]));
                            }
#pragma unroll
                            for (int k = 0; k < 16; ++k) pk[k] = pack_act<FP16>(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]));
                            const uint32_t at = into + (((2 * i + ((lane >> 3) & 1)) ^ ((lane >> 1) & 3)) << 4);   // 16-byte chunk of the row
#pragma unroll
                            for (int j = 0; j < 4; ++j) stmatrix_x4_trans(at + j * 16 * 64, pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
                        }
                        __syncwarp();
                        uint4 w[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) w[i] = ld_shared_v4(from + i * 8 * 64);   // row r0 + 8 i
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (8 * i < nrows) *reinterpret_cast<uint4*>(to + i * row8) = w[i];
                    } else {
                        // 32 queries at a time: their rounded values in the first 32 staging rows, the remainders in the others.
                        // (All 64 queries, one plane after the other, read dQ^T twice and kept it until the first plane had left:
                        // 1.68 -> 1.58 ms at B=2 S=8192 Hq=32 top-k 16 blocks without KL work.)
#pragma unroll 1
                        for (int y = 0; y < 2; ++y) {
#pragma unroll 1
                            for (int i = 0; i < 2; ++i) {
                                uint32_t v[16], hi[8], lo[8];
                                tmem_ld_16x256_x4(src + 32 * y + (static_cast<uint32_t>(16 * i) << 16), v);
                                tmem_ld_wait();
                                if (y + i == 2) {
                                    tc_fence_before_sync();
                                    warp_arrive(BAR(sm->dq_free[x]));
                                }
#pragma unroll
                                for (int k = 0; k < 8; ++k) {
                                    const float x0 = __uint_as_float(v[2 * k]), x1 = __uint_as_float(v[2 * k + 1]);
                                    hi[k] = pack_act<FP16>(x0, x1);
                                    lo[k] = pack_act<FP16>(x0 - act_lo<FP16>(hi[k]), x1 - act_hi<FP16>(hi[k]));
                                }
                                const uint32_t at = into + (((2 * i + ((lane >> 3) & 1)) ^ ((lane >> 1) & 3)) << 4);
#pragma unroll
                                for (int j = 0; j < 2; ++j) {
                                    stmatrix_x4_trans(at + j * 16 * 64, hi[4 * j], hi[4 * j + 1], hi[4 * j + 2], hi[4 * j + 3]);
                                    stmatrix_x4_trans(at + (32 + j * 16) * 64, lo[4 * j], lo[4 * j + 1], lo[4 * j + 2], lo[4 * j + 3]);
                                }
                            }
                            __syncwarp();
                            uint4 w[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) w[i] = ld_shared_v4(from + i * 8 * 64);
                            __nv_bfloat16* to2 = to + P.part_slots * P.mpp * kHeadDim;
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                if (32 * y + 8 * i < nrows) {
                                    *reinterpret_cast<uint4*>(to + i * row8) = w[i];
                                    *reinterpret_cast<uint4*>(to2 + i * row8) = w[4 + i];
                                }
                            to += 4 * row8;
                            __syncwarp();   // the rows have been read
                        }
                    }
                    warp_arrive(BAR(sm->ds_free[x]));
                }
                if (++hh == hpc) {
                    hh = 0;
                    ++chunk;
                }
            }
            if (!bad) {
                // sub-unit epilogue: add this sub-unit's share of dV_j and dK_j
                wait(BAR(sm->acc_full), nsub & 1, 3);
                if (!bad) {
                    tc_fence_after_sync();
                    const int64_t at = ((static_cast<int64_t>(ud.b) * P.Hkv + ud.kvh) * P.S + ud.j * kBlock) * kHeadDim;
#pragma unroll 1
                    for (int c = 0; c < 256; c += 32) {   // lane = key row of the block; columns 0..127 dV, 128..255 dK
                        float* drow = (c < 128 ? P.dv_acc : P.dk_acc) + at + static_cast<int64_t>(row) * kHeadDim + (c & 127);
                        uint32_t v[32];
                        tmem_ld32(tmem_addr(r2, quarter, c), v);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; i += 4)
                            red_add_v4(drow + i, __uint_as_float(v[i]), __uint_as_float(v[i + 1]), __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
                    }
                    tc_fence_before_sync();
                    warp_arrive(BAR(sm->acc_free));
                }
            }
        }
    } else {
        reg_inc<kBwdRegsCompute>();
        // =========================== compute groups ===========================
        // Both groups work on the same half tile, 32 queries each (group A 0..31, B 32..63 of the half): what counts is how soon
        // the operands of the half are written, because the products of the other half run meanwhile and no longer.
        // Thread = (key `row`, 32 queries of the half).  Reads S^T and dP^T, writes P^T and dS^T back into TMEM over S^T
        // (16 bit) and dS^T into the shared tile that feeds dQ^T = K^T dS^T.
        const int qoff = (warp >> 2) * 32;   // first query of the group inside a half
        const float2 sc2 = make_float2(P.scale_log2e, P.scale_log2e);
        // Sum over the main heads of P for this thread's 64 queries: the KL teacher, as packed fp16 pairs (values in [0,1], at
        // most Hq/Hp addends; what is formed from it is rounded to 16 bit anyway).  It goes to memory once per chunk.
        __half2 teacher[16], teacher_other[16];   // queries of this half, and of the other one: they change places after each
#pragma unroll
        for (int i = 0; i < 16; ++i) teacher[i] = teacher_other[i] = __floats2half2_rn(0.f, 0.f);
        UnitRec ud;
        for (uint32_t draw = 0; next_unit(draw, ud, std::integral_constant<int, kReads>{}); ++draw, ++nsub) {
            const int ntiles = (ud.chunk1 - ud.chunk0) * hpc;
            int hh = 0, chunk = ud.chunk0;
            for (int t = 0; t < ntiles && !bad; ++t, ++gt) {
                const uint32_t s = gt & 1;
                wait(BAR(sm->st_full[s]), (gt >> 1) & 1, 1);
                const BwdRowStats* st = &sm->stats[s];
                // only the first chunk of a reverse-index row can hold rows of the key block itself
                const bool own = (chunk == 0);
#pragma unroll 1
                for (int x = 0; x < 2; ++x) {
                    const int q0 = 64 * x + qoff;                     // first query of this thread inside the tile
                    const uint32_t rc = tmem + 128 * x + qoff;        // its first S^T column; dP^T is 64 columns on
                    const uint32_t ds_row = tile_ds + x * kPanelBytes + row * 128;
                    wait(BAR(sm->sdp_full[x]), gt & 1, 3);
                    // the half's panel of the dS^T tile doubles as the staging buffer of the previous tile's dQ store
                    if (gt >= 1) wait(BAR(sm->ds_free[x]), (gt - 1) & 1, 2);
                    if (bad) break;
                    tc_fence_after_sync();
                    const bool masked = own || (VARLEN && sm->any_low[s] != 0);
                    // Two instances of the body: the common tile must not pay for mask arithmetic.
                    auto compute_half = [&](auto masked_c) __attribute__((always_inline)) {
                        constexpr bool kMasked = decltype(masked_c)::value;
                        // Two pieces of 16 columns: the TMEM loads of the second are in flight while the first is worked on
                        // (tcgen05.wait::ld waits for every load issued so far, hence the order wait, issue, compute).
                        uint32_t sv[2][16], dv[2][16];
                        tmem_ld16(tmem_addr(rc, quarter, 0), sv[0]);
                        tmem_ld16(tmem_addr(rc, quarter, 64), dv[0]);
#pragma unroll
                        for (int cc = 0; cc < 2; ++cc) {
                            const int c = 16 * cc;
                            tmem_ld_wait();
                            if (cc == 0) {
                                tmem_ld16(tmem_addr(rc, quarter, 16), sv[1]);
                                tmem_ld16(tmem_addr(rc, quarter, 64 + 16), dv[1]);
                            }
                            uint32_t pk[8], dk[8];
#pragma unroll
                            for (int i4 = 0; i4 < 16; i4 += 4) {
                                const float4 nl4 = *reinterpret_cast<const float4*>(&st->neg_lse[q0 + c + i4]);
                                const float4 nd4 = *reinterpret_cast<const float4*>(&st->neg_delta[q0 + c + i4]);
                                uint32_t lim = 0x7f7f7f7fu, lw = 0u;
                                if (kMasked) {
                                    if (own) lim = *reinterpret_cast<const uint32_t*>(&st->limit[q0 + c + i4]);
                                    if (VARLEN) lw = *reinterpret_cast<const uint32_t*>(&st->low[q0 + c + i4]);
                                }
#pragma unroll
                                for (int i2 = 0; i2 < 4; i2 += 2) {
                                    const int i = i4 + i2;
                                    const float2 nl2 = i2 ? make_float2(nl4.z, nl4.w) : make_float2(nl4.x, nl4.y);
                                    const float2 a = f2_fma(f2_from_bits(sv[cc][i], sv[cc][i + 1]), sc2, nl2);   // log2 of the probability
                                    float p0 = fast_exp2(a.x);
                                    float p1 = fast_exp2(a.y);
                                    if (kMasked) {
                                        const int l0 = static_cast<int>((lim >> (8 * i2)) & 0xffu), l1 = static_cast<int>((lim >> (8 * i2 + 8)) & 0xffu);
                                        const int w0 = static_cast<int>((lw >> (8 * i2)) & 0xffu), w1 = static_cast<int>((lw >> (8 * i2 + 8)) & 0xffu);
                                        p0 = (row <= l0 && (!VARLEN || row >= w0)) ? p0 : 0.f;
                                        p1 = (row <= l1 && (!VARLEN || row >= w1)) ? p1 : 0.f;
                                    }
                                    // dS = P o (dP - delta)
                                    const float2 nd2 = i2 ? make_float2(nd4.z, nd4.w) : make_float2(nd4.x, nd4.y);
                                    const float2 d = f2_mul(make_float2(p0, p1), f2_add(f2_from_bits(dv[cc][i], dv[cc][i + 1]), nd2));
                                    pk[i >> 1] = pack_act<FP16>(p0, p1);
                                    dk[i >> 1] = pack_act<FP16>(d.x, d.y);
                                    if (KL) teacher[8 * cc + (i >> 1)] = __hadd2(teacher[8 * cc + (i >> 1)], __floats2half2_rn(p0, p1));
                                }
                            }
                            // 16-bit operands back into TMEM over the 16 score columns this thread has consumed: P^T, then dS^T,
                            // two queries per column.  dS^T also goes to the half's panel of the shared tile that feeds
                            // dQ^T = K^T dS^T (row = key, columns = queries).
                            tmem_st8(tmem_addr(rc, quarter, c), pk);
                            tmem_st8(tmem_addr(rc, quarter, c + 8), dk);
                            st_shared_v4(ds_row + ((2 * (qoff + c)) ^ ((row & 7) << 4)), dk[0], dk[1], dk[2], dk[3]);
                            st_shared_v4(ds_row + ((2 * (qoff + c) + 16) ^ ((row & 7) << 4)), dk[4], dk[5], dk[6], dk[7]);
                        }
                    };
                    if (masked) compute_half(std::true_type{});
                    else compute_half(std::false_type{});
                    tmem_st_wait();
                    fence_async_smem();
                    tc_fence_before_sync();
                    warp_arrive(BAR(sm->pds_full[x]));
                    if (KL) {
                        if (hh == hpc - 1) {
                            // Teacher of the chunk (layout: proxy_bwd.h)
                            const int64_t slot = ud.e0 - edge_base + static_cast<int64_t>(chunk) * kBlock + q0;
                            int left = ud.n - chunk * kBlock - q0;   // rows from this thread's first query on
                            uint32_t* dst = P.teacher + slot * 64;
#pragma unroll 1
                            for (int g8 = 0; g8 < 4; ++g8, left -= 8, dst += 512) {
                                if (left >= 8) {
                                    *reinterpret_cast<uint4*>(dst + 4 * row) = *reinterpret_cast<const uint4*>(&teacher[0]);
                                } else {
#pragma unroll
                                    for (int i = 0; i < 4; ++i) {
                                        if (2 * i + 1 < left) dst[i * 128 + row] = *reinterpret_cast<const uint32_t*>(&teacher[i]);
                                        else if (2 * i < left) reinterpret_cast<__half*>(dst + i * 128)[row] = __low2half(teacher[i]);
                                    }
                                }
#pragma unroll
                                for (int i = 0; i < 16; ++i) teacher[i] = i < 12 ? teacher[i + 4] : __floats2half2_rn(0.f, 0.f);
                            }
                        }
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const __half2 other = teacher[i];
                            teacher[i] = teacher_other[i];
                            teacher_other[i] = other;
                        }
                    }
                }
                if (bad) break;
                warp_arrive(BAR(sm->st_empty[s]));
                if (++hh == hpc) {
                    hh = 0;
                    ++chunk;
                }
            }
        }
    }
#ifdef FMSA_TRACE
    if (blockIdx.x == 0 && lane == 0) {
        trace_acc[0] = static_cast<unsigned long long>(clock64() - trace_t0);
        for (int i = 0; i < 8; ++i) g_bwd_trace[warp][i] = trace_acc[i];
    }
#endif
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

// -------------------------------------------------------------------------------------------
// dq[b,h,q,:] = sum over the row's edges of dq_part;  dq_proxy likewise, times the upstream
// gradient of kl_loss (a device scalar).  One warp per (batch*proxy head, query row).
// -------------------------------------------------------------------------------------------
struct BwdCombineParams {
    const __nv_bfloat16* dq_part;
    const __nv_bfloat16* dqp_part;
    const int32_t* edge_pos;   // sparse: [B*Hp, S, Kb]
    const int32_t* row_ptr;
    __nv_bfloat16* dq;         // (B,Hq,S,128) view: element strides below
    __nv_bfloat16* dqp;        // (B,Hp,S,128) view or null
    int32_t dq_sb, dq_sh, dq_ss, dqp_sb, dqp_sh, dqp_ss;   // element strides of the two views (each below 2^31)
    const float* grad_kl;      // device scalar or null (= 1)
    float scale, kl_out_scale; // factors the backward kernel left out of its partial rows
    int S, NB, Hq, Hp, mpp, ppk, Kb;
    int g_begin, G, dense;
    int hgroup;             // main heads per blockIdx.y
    int last_first;         // take the rows from the last one on
    int split;              // the partial buffers hold a second plane (rounding remainders) part_slots slots further on
    int64_t part_slots;
};

constexpr int64_t kLastFirstBytes = 512ll << 20;   // (figures: fmsa_sparse_bwd_combine)

// One sweep over the contiguous mpp*256-byte record of each edge; with more than eight main heads per proxy head blockIdx.y
// takes groups of heads, each a contiguous piece of the record (and group 0 the proxy row): at Hq/Hp = 12, 96 edges per row,
// two planes, B=1 S=16384 Hq=24, one head at a time with 8-byte loads took 4.26 ms, groups of six heads 2.48 ms.
template <int KITER, bool SPLIT, bool FP16, bool GROUPED>   // heads of a group <= 2*KITER: few accumulators, high occupancy (latency bound)
__global__ void __launch_bounds__(256, (KITER <= 2) ? 4 : 2) bwd_combine_kernel(const BwdCombineParams P) {
    wait_for_previous_kernel();
    const int lane = threadIdx.x & 31;
    const int64_t w = static_cast<int64_t>(P.last_first ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * 8 + (threadIdx.x >> 5);
    const int64_t bp0 = static_cast<int64_t>(P.g_begin) * P.ppk;
    if (w >= static_cast<int64_t>(P.G) * P.ppk * P.S) return;
    const int64_t bp = bp0 + w / P.S;
    const int q = static_cast<int>(w % P.S);
    const int b = static_cast<int>(bp / P.Hp), p = static_cast<int>(bp % P.Hp);
    const int64_t edge_base = P.dense ? dense_edge_base(bp0, P.S, P.NB) : static_cast<int64_t>(P.row_ptr[bp0 * P.NB]);
    const int nslots = P.dense ? (q >> 7) + 1 : P.Kb;
    const int32_t* erow = P.dense ? nullptr : P.edge_pos + (bp * P.S + q) * P.Kb;
    auto slot_of = [&](int s) -> int64_t {
        if (s >= nslots) return -1;
        if (P.dense) return dense_edge_base(bp, P.S, P.NB) + dense_row_offset(s, P.S) + (q - s * kBlock) - edge_base;
        const int e = erow[s];
        return e < 0 ? -1 : static_cast<int64_t>(e) - edge_base;
    };
    const int h0 = GROUPED ? blockIdx.y * P.hgroup : 0, hn = GROUPED ? min(P.hgroup, P.mpp - h0) : P.mpp;   // this block's main heads
    const int nchunk = hn * 16;
    float acc[KITER][8];
#pragma unroll
    for (int k = 0; k < KITER; ++k)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[k][e] = 0.f;
    float pa0 = 0.f, pa1 = 0.f, pa2 = 0.f, pa3 = 0.f;   // proxy row: lane owns columns 4*lane..+3
    // Four edges at a time: every load of the group is issued before the first sum (the kernel is bound by memory
    // latency; left to itself the compiler batches the loads only when the register budget happens to allow it).
    const bool has_proxy = P.dqp != nullptr && (!GROUPED || blockIdx.y == 0);
    for (int s0 = 0; s0 < nslots; s0 += 32) {
        const int sl = static_cast<int>(slot_of(s0 + lane));   // slot numbers of a pass fit 31 bits
        const int cnt = min(32, nslots - s0);
        for (int i = 0; i < cnt; i += 4) {
            int si[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int v = __shfl_sync(0xffffffffu, sl, (i + u) & 31);
                si[u] = (i + u < cnt) ? v : -1;
            }
#pragma unroll
            for (int part = 0; part < (SPLIT ? 2 : 1); ++part) {
                uint4 raw[4][KITER];
                uint2 praw[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int64_t sp = static_cast<int64_t>(si[u]) + part * P.part_slots;
                    const __nv_bfloat16* rec = P.dq_part + (sp * P.mpp + h0) * kHeadDim;
#pragma unroll
                    for (int k = 0; k < KITER; ++k) {
                        const int ck = k * 32 + lane;
                        raw[u][k] = (si[u] >= 0 && ck < nchunk) ? *reinterpret_cast<const uint4*>(rec + ck * 8) : make_uint4(0, 0, 0, 0);
                    }
                    praw[u] = (si[u] >= 0 && has_proxy) ? *reinterpret_cast<const uint2*>(P.dqp_part + sp * kHeadDim + lane * 4)
                                                        : make_uint2(0, 0);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
#pragma unroll
                    for (int k = 0; k < KITER; ++k) {
                        const uint32_t w4[4] = {raw[u][k].x, raw[u][k].y, raw[u][k].z, raw[u][k].w};
                        if constexpr (KITER >= 3) {   // packed adds pay at 120-128 registers and two CTAs per SM, not at 64
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const float2 a = f2_add(make_float2(acc[k][2 * e], acc[k][2 * e + 1]),
                                                        make_float2(act_lo<FP16>(w4[e]), act_hi<FP16>(w4[e])));
                                acc[k][2 * e] = a.x;
                                acc[k][2 * e + 1] = a.y;
                            }
                        } else {
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                acc[k][2 * e] += act_lo<FP16>(w4[e]);
                                acc[k][2 * e + 1] += act_hi<FP16>(w4[e]);
                            }
                        }
                    }
                    pa0 += act_lo<FP16>(praw[u].x);
                    pa1 += act_hi<FP16>(praw[u].x);
                    pa2 += act_lo<FP16>(praw[u].y);
                    pa3 += act_hi<FP16>(praw[u].y);
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < KITER; ++k) {
        const int ck = k * 32 + lane;
        if (ck < nchunk) {
            const int hh = h0 + (ck >> 4), col = (ck & 15) * 8;
            uint4 o;
            o.x = pack_act<FP16>(acc[k][0] * P.scale, acc[k][1] * P.scale);
            o.y = pack_act<FP16>(acc[k][2] * P.scale, acc[k][3] * P.scale);
            o.z = pack_act<FP16>(acc[k][4] * P.scale, acc[k][5] * P.scale);
            o.w = pack_act<FP16>(acc[k][6] * P.scale, acc[k][7] * P.scale);
            *reinterpret_cast<uint4*>(P.dq + (static_cast<int64_t>(b) * P.dq_sb + static_cast<int64_t>(p * P.mpp + hh) * P.dq_sh + static_cast<int64_t>(q) * P.dq_ss) + col) = o;
        }
    }
    if (has_proxy) {
        const float gk = (P.grad_kl ? *P.grad_kl : 1.f) * P.kl_out_scale;
        uint2 o;
        o.x = pack_act<FP16>(pa0 * gk, pa1 * gk);
        o.y = pack_act<FP16>(pa2 * gk, pa3 * gk);
        *reinterpret_cast<uint2*>(P.dqp + (static_cast<int64_t>(b) * P.dqp_sb + static_cast<int64_t>(p) * P.dqp_sh + static_cast<int64_t>(q) * P.dqp_ss) + lane * 4) = o;
    }
}

// -------------------------------------------------------------------------------------------
// delta[b,h,q] = sum_d out[b,q,h,d] * dout[b,q,h,d]   (flash_msa/flash_msa.py:99)
// -------------------------------------------------------------------------------------------
// One CTA per (batch, 8 consecutive query positions): half-warp g takes position g%8 and every other group of four heads,
// each lane reading 16 bytes of the `out` row and of the `dout` row (a half-warp covers one 256-byte row per load, four
// rows in flight); the sums meet in shared memory so that delta leaves in 32-byte runs along the sequence.  Bound by memory;
// with 32 positions per CTA there were too few CTAs to hide its latency (B=3 S=1664 Hq=20:
// 27.9 -> 9.6 us; B=2 S=8192 Hq=32: 52.6 -> 46.9 us).
// `zero`: 16-byte words to clear on the way, the gradients' accumulators of a whole pass (their memset stood between two kernels:
// a pass of B=3 S=1664 Hq=20 261.4 -> 259.1 us, of B=2 S=8192 Hq=32 3600 -> 3590, back to back).
template <bool FP16>
__global__ void __launch_bounds__(256) delta_kernel(const __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ dout,
                                                    int64_t do_sb, int64_t do_ss, int64_t do_sh, float* __restrict__ delta,
                                                    int B, int S, int Hq, uint4* __restrict__ zero, int64_t nzero) {
    wait_for_previous_kernel();
    extern __shared__ float sdelta[];   // [Hq][8]
    const int lane = threadIdx.x & 31, l16 = lane & 15;
    const int g = threadIdx.x >> 4;   // half-warp 0..15
    const int qblocks = S >> 3;
    const int b = blockIdx.x / qblocks, q0 = (blockIdx.x % qblocks) << 3;
    auto dot8 = [](const uint4& a, const uint4& d) {
        return act_lo<FP16>(a.x) * act_lo<FP16>(d.x) + act_hi<FP16>(a.x) * act_hi<FP16>(d.x) + act_lo<FP16>(a.y) * act_lo<FP16>(d.y) +
               act_hi<FP16>(a.y) * act_hi<FP16>(d.y) + act_lo<FP16>(a.z) * act_lo<FP16>(d.z) + act_hi<FP16>(a.z) * act_hi<FP16>(d.z) +
               act_lo<FP16>(a.w) * act_lo<FP16>(d.w) + act_hi<FP16>(a.w) * act_hi<FP16>(d.w);
    };
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; i < nzero; i += static_cast<int64_t>(gridDim.x) * 256)
        zero[i] = make_uint4(0u, 0u, 0u, 0u);
    const int ql = g & 7, q = q0 + ql;
    const __nv_bfloat16* orow = out + (static_cast<int64_t>(b) * S + q) * Hq * kHeadDim + l16 * 8;
    const __nv_bfloat16* drow = dout + b * do_sb + q * do_ss + l16 * 8;
    for (int h = 4 * (g >> 3); h < Hq; h += 8) {
        uint4 a[4], d[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int hi = min(h + i, Hq - 1);
            a[i] = *reinterpret_cast<const uint4*>(orow + static_cast<int64_t>(hi) * kHeadDim);
            d[i] = *reinterpret_cast<const uint4*>(drow + hi * do_sh);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float sum = dot8(a[i], d[i]);
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
            if (l16 == 0 && h + i < Hq) sdelta[(h + i) * 8 + ql] = sum;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < Hq * 8; i += 256) delta[(static_cast<int64_t>(b) * Hq + (i >> 3)) * S + q0 + (i & 7)] = sdelta[i];
}

// dst = bf16(src * const_scale * factor), factor = *scale_ptr when given (the upstream kl gradient lives on the
// device: flash_msa/flash_msa.py:122-125) else 1.
template <bool FP16>
__global__ void __launch_bounds__(256) cast_scaled_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, int64_t n4,
                                                          const float* __restrict__ scale_ptr, float const_scale) {
    const float f = (scale_ptr ? *scale_ptr : 1.f) * const_scale;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4; i += stride) {
        const float4 v = reinterpret_cast<const float4*>(src)[i];
        uint2 o;
        o.x = pack_act<FP16>(v.x * f, v.y * f);
        o.y = pack_act<FP16>(v.z * f, v.w * f);
        reinterpret_cast<uint2*>(dst)[i] = o;
    }
}

// The same cast with a strided destination: src is contiguous fp32 [B,H,S,128], dst a (B,H,S,128) view given by
// element strides (a gradient written straight into (B,S,H,128) storage).  One thread per four elements.
template <bool FP16>
__global__ void __launch_bounds__(256) cast_scaled_rows_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst,
                                                               int64_t sb, int64_t sh, int64_t ss, int H, int S, int64_t n4,
                                                               const float* __restrict__ scale_ptr, float const_scale) {
    const float f = (scale_ptr ? *scale_ptr : 1.f) * const_scale;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4; i += stride) {
        const int64_t rowi = i >> 5;                // 32 float4 per row of 128
        const int c4 = static_cast<int>(i & 31);
        const int sq = static_cast<int>(rowi % S);
        const int64_t bh = rowi / S;
        const int h = static_cast<int>(bh % H);
        const int64_t b = bh / H;
        const float4 v = reinterpret_cast<const float4*>(src)[i];
        uint2 o;
        o.x = pack_act<FP16>(v.x * f, v.y * f);
        o.y = pack_act<FP16>(v.z * f, v.w * f);
        *reinterpret_cast<uint2*>(dst + b * sb + h * sh + sq * ss + c4 * 4) = o;
    }
}

// dsinks[h] = -sum over the rows of head h of exp(sink_h - lse') * delta: one CTA per head, in a fixed order.
__global__ void __launch_bounds__(512) sink_grad_kernel(const float* __restrict__ lse, const float* __restrict__ delta,
                                                        const float* __restrict__ sinks, float* __restrict__ dsinks, int B, int S, int Hq) {
    wait_for_previous_kernel();
    __shared__ float part[16];
    const int h = blockIdx.x;
    const float sk = sinks[h];
    float sum = 0.f;
    for (int b = 0; b < B; ++b) {
        const int64_t at = (static_cast<int64_t>(b) * Hq + h) * S;
        for (int s = threadIdx.x; s < S; s += 512) sum += expf(sk - lse[at + s]) * delta[at + s];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        float total = 0.f;
        for (int i = 0; i < 16; ++i) total += part[i];
        dsinks[h] = -total;
    }
}

// dK, dV and dKp from their fp32 accumulators in one launch (blockIdx.y): 8 elements per thread into (B,H,S,128) views.
template <bool FP16>
__global__ void __launch_bounds__(256) cast_grads_kernel(const CastJobs J) {
    wait_for_previous_kernel();
    const CastJob& c = J.job[blockIdx.y];
    const float f = (c.factor ? *c.factor : 1.f) * c.scale;
    const uint32_t n8 = c.n8, stride = gridDim.x * 256;
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < n8; i += stride) {
        const uint32_t rowi = i >> 4, c8 = (i & 15) * 8;
        const uint32_t bh = rowi / J.S, sq = rowi - bh * J.S, b = bh / c.H, h = bh - b * c.H;
        const float4 v0 = reinterpret_cast<const float4*>(c.src)[2 * static_cast<int64_t>(i)];
        const float4 v1 = reinterpret_cast<const float4*>(c.src)[2 * static_cast<int64_t>(i) + 1];
        uint4 o;
        o.x = pack_act<FP16>(v0.x * f, v0.y * f);
        o.y = pack_act<FP16>(v0.z * f, v0.w * f);
        o.z = pack_act<FP16>(v1.x * f, v1.y * f);
        o.w = pack_act<FP16>(v1.z * f, v1.w * f);
        *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(c.dst) + b * c.sb + h * c.sh + sq * c.ss + c8) = o;
    }
}

}  // namespace

int launch_cast_grads(const CastJobs& jobs, int count, bool fp16, cudaStream_t st) {
    uint32_t most = 0;
    for (int i = 0; i < count; ++i) most = jobs.job[i].n8 > most ? jobs.job[i].n8 : most;
    uint32_t grid = (most + 255) / 256;
    if (grid > 148 * 8) grid = 148 * 8;
    const dim3 g(grid, static_cast<unsigned>(count));
    launch_chained(fp16 ? cast_grads_kernel<true> : cast_grads_kernel<false>, g, 256, 0, st, jobs);
    return check_launch();
}

int launch_sink_grad(const float* lse, const float* delta, const float* sinks, float* dsinks, int B, int S, int Hq, cudaStream_t st) {
    launch_chained(sink_grad_kernel, Hq, 512, 0, st, lse, delta, sinks, dsinks, B, S, Hq);
    return check_launch();
}

}  // namespace fmsa

extern "C" int fmsa_cast_scaled_rows(const float* src, const fmsa_tensor* dst, int32_t B, int32_t H, int32_t S,
                                     const float* scale_ptr, float const_scale, int32_t dtype, void* stream) {
    using namespace fmsa;
    FMSA_REQUIRE(src && dst && dst->ptr && B > 0 && H > 0 && S > 0);
    FMSA_REQUIRE(dtype == FMSA_DTYPE_BF16 || dtype == FMSA_DTYPE_FP16);
    FMSA_REQUIRE(aligned16(src) && (reinterpret_cast<uintptr_t>(dst->ptr) & 7u) == 0);
    FMSA_REQUIRE(dst->stride_b % 4 == 0 && dst->stride_h % 4 == 0 && dst->stride_s % 4 == 0);
    const int64_t n4 = static_cast<int64_t>(B) * H * S * (kHeadDim / 4);
    int64_t grid = (n4 + 255) / 256;
    if (grid > 148 * 16) grid = 148 * 16;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == FMSA_DTYPE_FP16)
        cast_scaled_rows_kernel<true><<<static_cast<unsigned>(grid), 256, 0, st>>>(
            src, static_cast<__nv_bfloat16*>(const_cast<void*>(dst->ptr)), dst->stride_b, dst->stride_h, dst->stride_s, H, S, n4, scale_ptr, const_scale);
    else
        cast_scaled_rows_kernel<false><<<static_cast<unsigned>(grid), 256, 0, st>>>(
            src, static_cast<__nv_bfloat16*>(const_cast<void*>(dst->ptr)), dst->stride_b, dst->stride_h, dst->stride_s, H, S, n4, scale_ptr, const_scale);
    return check_launch();
}

extern "C" int fmsa_bwd_delta(const void* out, const fmsa_tensor* d_out, float* delta, int32_t B, int32_t S, int32_t Hq,
                              int32_t dtype, void* stream) {
    return fmsa::launch_delta(out, d_out, delta, B, S, Hq, dtype, nullptr, 0, static_cast<cudaStream_t>(stream));
}

int fmsa::launch_delta(const void* out, const fmsa_tensor* d_out, float* delta, int B, int S, int Hq, int dtype, void* zero, int64_t zero_bytes,
                       cudaStream_t st) {
    using namespace fmsa;
    FMSA_REQUIRE(out && d_out && d_out->ptr && delta && B > 0 && S > 0 && Hq > 0);
    FMSA_REQUIRE(dtype == FMSA_DTYPE_BF16 || dtype == FMSA_DTYPE_FP16);
    FMSA_REQUIRE(aligned16(out) && aligned16(d_out->ptr));
    FMSA_REQUIRE(d_out->stride_b % 8 == 0 && d_out->stride_h % 8 == 0 && d_out->stride_s % 8 == 0);
    const int64_t grid = static_cast<int64_t>(B) * (S / 8);
    FMSA_REQUIRE(S % 32 == 0 && grid <= 0x7fffffffLL && Hq * 8 * sizeof(float) <= 48 * 1024);
    const size_t smem = static_cast<size_t>(Hq) * 8 * sizeof(float);
    launch_chained(dtype == FMSA_DTYPE_FP16 ? delta_kernel<true> : delta_kernel<false>, static_cast<unsigned>(grid), 256, smem,
                   st, static_cast<const __nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(d_out->ptr),
                   d_out->stride_b, d_out->stride_s, d_out->stride_h, delta, B, S, Hq, static_cast<uint4*>(zero), zero_bytes / 16);
    return check_launch();
}

extern "C" int fmsa_cast_scaled(const float* src, void* dst, int64_t n, const float* scale_ptr, float const_scale,
                                int32_t dtype, void* stream) {
    using namespace fmsa;
    FMSA_REQUIRE(src && dst && n >= 0 && n % 4 == 0);
    FMSA_REQUIRE(dtype == FMSA_DTYPE_BF16 || dtype == FMSA_DTYPE_FP16);
    FMSA_REQUIRE(aligned16(src) && (reinterpret_cast<uintptr_t>(dst) & 7u) == 0);
    if (n == 0) return FMSA_OK;
    const int64_t n4 = n / 4;
    int64_t grid = (n4 + 255) / 256;
    if (grid > 148 * 16) grid = 148 * 16;
    if (dtype == FMSA_DTYPE_FP16)
        cast_scaled_kernel<true><<<static_cast<unsigned>(grid), 256, 0, static_cast<cudaStream_t>(stream)>>>(
            src, static_cast<__nv_bfloat16*>(dst), n4, scale_ptr, const_scale);
    else
        cast_scaled_kernel<false><<<static_cast<unsigned>(grid), 256, 0, static_cast<cudaStream_t>(stream)>>>(
            src, static_cast<__nv_bfloat16*>(dst), n4, scale_ptr, const_scale);
    return check_launch();
}

extern "C" int fmsa_sparse_bwd(const fmsa_problem* pb, const fmsa_tensor* q, const fmsa_tensor* k, const fmsa_tensor* v,
                               const fmsa_tensor* q_proxy, const fmsa_tensor* k_proxy, const fmsa_tensor* d_out,
                               const float* lse, const float* lse_proxy, const float* delta, const int32_t* row_ptr,
                               const int32_t* col_q, void* dq_part, void* dqp_part, int64_t part_slots, int32_t split,
                               float* dkp_acc, float* dk_acc, float* dv_acc, int32_t g_begin, int32_t g_count, int32_t with_kl,
                               int32_t dense, float* kl_value, int32_t* counter, int32_t* status, void* stream) {
    return fmsa::launch_sparse_bwd(pb, q, k, v, q_proxy, k_proxy, d_out, lse, lse_proxy, delta, row_ptr, col_q, dq_part, dqp_part,
                                   part_slots, split, dkp_acc, dk_acc, dv_acc, g_begin, g_count, with_kl, dense, kl_value, counter,
                                   counter, true, status, static_cast<cudaStream_t>(stream));
}

int fmsa::launch_sparse_bwd(const fmsa_problem* pb, const fmsa_tensor* q, const fmsa_tensor* k, const fmsa_tensor* v,
                            const fmsa_tensor* q_proxy, const fmsa_tensor* k_proxy, const fmsa_tensor* d_out, const float* lse,
                            const float* lse_proxy, const float* delta, const int32_t* row_ptr, const int32_t* col_q, void* dq_part,
                            void* dqp_part, int64_t part_slots, int split, float* dkp_acc, float* dk_acc, float* dv_acc, int g_begin,
                            int g_count, int with_kl, int dense, float* kl_value, int32_t* counter, int32_t* counter_proxy,
                            bool zero_counters, int32_t* status, cudaStream_t st) {
    using namespace fmsa;
    FMSA_REQUIRE(problem_ok(pb));
    FMSA_REQUIRE(q && k && v && d_out && q->ptr && k->ptr && v->ptr && d_out->ptr);
    FMSA_REQUIRE(lse && delta && dq_part && dk_acc && dv_acc && counter && status);
    FMSA_REQUIRE(dense || (row_ptr && col_q));
    FMSA_REQUIRE(!with_kl || (q_proxy && k_proxy && q_proxy->ptr && k_proxy->ptr && lse_proxy && dqp_part && dkp_acc));
    FMSA_REQUIRE(g_begin >= 0 && g_count > 0 && g_begin + g_count <= pb->B * pb->Hkv);
    FMSA_REQUIRE(dense || (pb->top_k_blocks >= 1 && pb->top_k_blocks <= pb->S / kBlock));
    FMSA_REQUIRE(pb->scale > 0.f);
    FMSA_REQUIRE(static_cast<int64_t>(pb->B) * pb->Hp <= 65535 && pb->S / kBlock <= 32767);   // 16-bit fields of the sub-unit record
    if (part_slots < fmsa_fwd_partial_slots(pb, g_count, dense)) return FMSA_ERR_WORKSPACE;
    FMSA_REQUIRE(tma_compatible(k->ptr, k->stride_b, k->stride_h, k->stride_s));
    FMSA_REQUIRE(tma_compatible(v->ptr, v->stride_b, v->stride_h, v->stride_s));
    FMSA_REQUIRE(tma_compatible(q->ptr, q->stride_b, q->stride_h, q->stride_s));
    FMSA_REQUIRE(tma_compatible(d_out->ptr, d_out->stride_b, d_out->stride_h, d_out->stride_s));
    if (with_kl) {
        FMSA_REQUIRE(tma_compatible(q_proxy->ptr, q_proxy->stride_b, q_proxy->stride_h, q_proxy->stride_s));
        FMSA_REQUIRE(tma_compatible(k_proxy->ptr, k_proxy->stride_b, k_proxy->stride_h, k_proxy->stride_s));
    }
    FMSA_REQUIRE(aligned16(dk_acc) && aligned16(dv_acc) && (!with_kl || aligned16(dkp_acc)));
    FMSA_REQUIRE(aligned16(dq_part) && (!with_kl || aligned16(dqp_part)));
    FMSA_REQUIRE(gather_compatible(q->ptr, q->stride_b, q->stride_h, q->stride_s));
    FMSA_REQUIRE(gather_compatible(d_out->ptr, d_out->stride_b, d_out->stride_h, d_out->stride_s));
    if (with_kl) FMSA_REQUIRE(gather_compatible(q_proxy->ptr, q_proxy->stride_b, q_proxy->stride_h, q_proxy->stride_s));
    FMSA_REQUIRE(part_slots > 0 && part_slots * (split ? 2 : 1) < 0x7fffffffLL);
    const uint64_t q_rows = gather_rows(pb->B, pb->Hq, pb->S, q->stride_b, q->stride_h, q->stride_s);
    const uint64_t do_rows = gather_rows(pb->B, pb->Hq, pb->S, d_out->stride_b, d_out->stride_h, d_out->stride_s);
    CUtensorMap tq, tdo, tk, tv;
    if (!make_tmap_gather(&tq, q->ptr, q_rows) || !make_tmap_gather(&tdo, d_out->ptr, do_rows) ||
        !make_tmap_bhsd(&tk, k->ptr, pb->B, pb->Hkv, pb->S, k->stride_b, k->stride_h, k->stride_s, 128) ||
        !make_tmap_bhsd(&tv, v->ptr, pb->B, pb->Hkv, pb->S, v->stride_b, v->stride_h, v->stride_s, 128))
        return FMSA_ERR_CUDA;

    BwdParams P;
    P.q_row_b = static_cast<int32_t>(q->stride_b / 128); P.q_row_h = static_cast<int32_t>(q->stride_h / 128); P.q_row_s = static_cast<int32_t>(q->stride_s / 128);
    P.do_row_b = static_cast<int32_t>(d_out->stride_b / 128); P.do_row_h = static_cast<int32_t>(d_out->stride_h / 128); P.do_row_s = static_cast<int32_t>(d_out->stride_s / 128);
    P.q_rows_total = static_cast<int32_t>(q_rows); P.do_rows_total = static_cast<int32_t>(do_rows);
    P.lse = lse; P.delta = delta;
    P.col_q = col_q; P.doc_start = pb->doc_start;
    P.dq_part = static_cast<__nv_bfloat16*>(dq_part); P.teacher = static_cast<uint32_t*>(dqp_part);
    P.part_slots = part_slots;
    P.dk_acc = dk_acc; P.dv_acc = dv_acc;
    P.status = status;
    P.S = pb->S; P.Hq = pb->Hq; P.Hkv = pb->Hkv; P.mpp = pb->Hq / pb->Hp;
    P.scale_log2e = pb->scale * kLog2e;

    const int sms = device_sm_count();
    const bool fp16 = pb->dtype == FMSA_DTYPE_FP16;
    const bool varlen = P.doc_start != nullptr;
    using KernelFn = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, BwdParams);
#define FMSA_BWD_KERNELS(F, V) \
    sparse_bwd_kernel<F, V, false, false>, sparse_bwd_kernel<F, V, false, true>, sparse_bwd_kernel<F, V, true, false>, sparse_bwd_kernel<F, V, true, true>
    static const KernelFn kernels[16] = {FMSA_BWD_KERNELS(false, false), FMSA_BWD_KERNELS(false, true), FMSA_BWD_KERNELS(true, false),
                                         FMSA_BWD_KERNELS(true, true)};
#undef FMSA_BWD_KERNELS
    const KernelFn kernel = kernels[(fp16 ? 8 : 0) + (varlen ? 4 : 0) + (with_kl ? 2 : 0) + (split ? 1 : 0)];
    const void* kfn = reinterpret_cast<const void*>(kernel);
    if (sms <= 0 || !ensure_smem_attr(kfn, kBwdSmemBytes)) return FMSA_ERR_CUDA;
    if (zero_counters && cudaMemsetAsync(counter, 0, sizeof(int32_t), st) != cudaSuccess) return FMSA_ERR_CUDA;
    UnitSpace& U = P.units;
    U.row_ptr = row_ptr; U.counter = counter;
    U.S = pb->S; U.NB = pb->S / kBlock; U.Hkv = pb->Hkv; U.Hp = pb->Hp; U.ppk = pb->Hp / pb->Hkv;
    U.g_begin = g_begin; U.dense = dense ? 1 : 0;
    FMSA_REQUIRE(enumerate_subunits(&U.sub, fmsa_fwd_partial_slots(pb, g_count, dense), g_count, U.NB, U.NB, U.ppk, sms));
    const int grid = U.sub.n < sms ? U.sub.n : sms;
    launch_chained(kernel, grid, kBwdThreads, kBwdSmemBytes, st, tq, tdo, tk, tv, P);
    if (with_kl) {
        if (zero_counters && cudaMemsetAsync(counter_proxy, 0, sizeof(int32_t), st) != cudaSuccess) return FMSA_ERR_CUDA;
        U.counter = counter_proxy;
        const int rc = launch_proxy_bwd(pb, *q_proxy, *k_proxy, lse_proxy, U, col_q, dqp_part, part_slots, split, dkp_acc, kl_value, grid, status, st);
        if (rc != FMSA_OK) return rc;
    }
    return check_launch();
}

extern "C" int fmsa_sparse_bwd_combine(const fmsa_problem* pb, const void* dq_part, const void* dqp_part,
                                       int64_t part_slots, int32_t split, const int32_t* edge_pos, const int32_t* row_ptr,
                                       const fmsa_tensor* dq, const fmsa_tensor* dq_proxy, const float* grad_kl,
                                       int32_t g_begin, int32_t g_count, int32_t dense, void* stream) {
    using namespace fmsa;
    FMSA_REQUIRE(problem_ok(pb));
    FMSA_REQUIRE(dq_part && dq && dq->ptr);
    FMSA_REQUIRE(dense || (edge_pos && row_ptr));
    FMSA_REQUIRE(!dq_proxy || (dq_proxy->ptr && dqp_part));
    FMSA_REQUIRE(aligned16(dq->ptr) && dq->stride_b % 8 == 0 && dq->stride_h % 8 == 0 && dq->stride_s % 8 == 0);
    FMSA_REQUIRE(!dq_proxy || (aligned16(dq_proxy->ptr) && dq_proxy->stride_b % 8 == 0 && dq_proxy->stride_h % 8 == 0 &&
                               dq_proxy->stride_s % 8 == 0));
    FMSA_REQUIRE(g_begin >= 0 && g_count > 0 && g_begin + g_count <= pb->B * pb->Hkv);
    FMSA_REQUIRE(!split || part_slots > 0);
    BwdCombineParams P;
    P.dq_part = static_cast<const __nv_bfloat16*>(dq_part); P.dqp_part = static_cast<const __nv_bfloat16*>(dqp_part);
    P.edge_pos = edge_pos; P.row_ptr = row_ptr;
    P.split = split ? 1 : 0; P.part_slots = part_slots;
    auto fits = [](int64_t x) { return x >= 0 && x < 0x7fffffffLL; };
    FMSA_REQUIRE(fits(dq->stride_b) && fits(dq->stride_h) && fits(dq->stride_s));
    FMSA_REQUIRE(!dq_proxy || (fits(dq_proxy->stride_b) && fits(dq_proxy->stride_h) && fits(dq_proxy->stride_s)));
    P.dq = static_cast<__nv_bfloat16*>(const_cast<void*>(dq->ptr));
    P.dq_sb = static_cast<int32_t>(dq->stride_b); P.dq_sh = static_cast<int32_t>(dq->stride_h); P.dq_ss = static_cast<int32_t>(dq->stride_s);
    P.dqp = dq_proxy ? static_cast<__nv_bfloat16*>(const_cast<void*>(dq_proxy->ptr)) : nullptr;
    P.dqp_sb = dq_proxy ? static_cast<int32_t>(dq_proxy->stride_b) : 0; P.dqp_sh = dq_proxy ? static_cast<int32_t>(dq_proxy->stride_h) : 0;
    P.dqp_ss = dq_proxy ? static_cast<int32_t>(dq_proxy->stride_s) : 0;
    P.grad_kl = grad_kl;
    P.S = pb->S; P.NB = pb->S / kBlock; P.Hq = pb->Hq; P.Hp = pb->Hp; P.mpp = pb->Hq / pb->Hp; P.ppk = pb->Hp / pb->Hkv;
    P.Kb = pb->top_k_blocks; P.g_begin = g_begin; P.G = g_count; P.dense = dense ? 1 : 0;
    P.scale = pb->scale;
    P.kl_out_scale = pb->scale / (static_cast<float>(pb->B) * pb->Hp * pb->S);
    const int64_t rows = static_cast<int64_t>(g_count) * P.ppk * P.S;
    const int64_t grid = (rows + 7) / 8;
    FMSA_REQUIRE(grid <= 0x7fffffffLL);
    // Up to a few times L2 (126 MB) a good part of the partial rows, those written last, is still there.  B=1 Hq=16 Hp=4 top-k 16 blocks, one
    // plane: 160 MB 29.2 -> 27.1 us, 240 MB 45.6 -> 42.4, 320 MB 59.9 -> 57.9, 480 MB 88.6 both ways; top-k 4: 160 MB 47.5 -> 45.5, 320 MB 84.4 ->
    // 82.4, 480 MB 119.3 -> 117.2.  From there to 1.3 GB the two orders are within 1 to 3 %, of 5 GB in two planes too little is left and the other
    // order is the faster one (B=1 S=16384 top-k 96: 2.53 -> 2.61 ms), so the line is at the end of the clear gain.
    const int64_t part_bytes = fmsa_fwd_partial_slots(pb, g_count, dense) * (P.mpp + (dq_proxy ? 1 : 0)) * kHeadDim * 2 * (split ? 2 : 1);
    P.last_first = part_bytes <= kLastFirstBytes ? 1 : 0;
    const int groups = P.mpp <= 8 ? 1 : (P.mpp + 5) / 6;   // as in the forward combine
    P.hgroup = (P.mpp + groups - 1) / groups;
    const dim3 cg(static_cast<unsigned>(grid), static_cast<unsigned>(groups));
    cudaStream_t cst = static_cast<cudaStream_t>(stream);
    const bool fp16 = pb->dtype == FMSA_DTYPE_FP16;
#define FMSA_BWD_COMBINE(K, G)                                                                          \
    do {                                                                                             \
        if (fp16) {                                                                                  \
            if (P.split) launch_chained(bwd_combine_kernel<K, true, true, G>, cg, 256, 0, cst, P); \
            else launch_chained(bwd_combine_kernel<K, false, true, G>, cg, 256, 0, cst, P); \
        } else {                                                                                     \
            if (P.split) launch_chained(bwd_combine_kernel<K, true, false, G>, cg, 256, 0, cst, P); \
            else launch_chained(bwd_combine_kernel<K, false, false, G>, cg, 256, 0, cst, P); \
        }                                                                                            \
    } while (0)
    if (groups > 1) FMSA_BWD_COMBINE(3, true);
    else if (P.mpp <= 2) FMSA_BWD_COMBINE(1, false);
    else if (P.mpp <= 4) FMSA_BWD_COMBINE(2, false);
    else if (P.mpp <= 6) FMSA_BWD_COMBINE(3, false);
    else FMSA_BWD_COMBINE(4, false);
#undef FMSA_BWD_COMBINE
    return check_launch();
}

#ifdef FMSA_TRACE
extern "C" int fmsa_debug_bwd_trace(unsigned long long* host_out) {
    return cudaMemcpyFromSymbol(host_out, fmsa::g_bwd_trace, sizeof(unsigned long long) * 20 * 8) == cudaSuccess ? 0 : -4;
}
#endif

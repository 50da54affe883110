// Query-tile stationary forward for query tiles that select most of the key blocks they can see.
//
// The key-block stationary forward (sparse_fwd.cu) pays for every edge (query row, key block) with a partial row that is
// written, read again and merged; in exchange it never multiplies a row with a block it did not select.  A query tile
// whose rows select most of its causal blocks has little to gain from that: walking all blocks that any of its 128 rows selected
// keeps the row's output in TMEM from the first block to the last, and nothing but `out` and the log-sum-exp leaves the SM.
// This is the forward of the first query tiles of a sparse call (which those are: forward_tiles in msa_common.cuh) and of every tile
// of a dense one.  Same numerics as before except that the sum over the blocks is fp32 throughout (no 16-bit partial rows).
//
// Work item = (batch, query tile, main head), or (batch, query tile, proxy head), which needs the log-sum-exp only.  Persistent CTAs
// draw items from a global counter, longest first.  A step of an item is one visited block: S = Q K_j^T into one of three S buffers in
// TMEM, P = exp2(S*c - m) over it (16 bit), O += P V_j in the lanes of the rows that selected the block (leaving the others' lanes out,
// instead of multiplying zeros, keeps a value that is not finite away from them).  Roles (warp index): 0-3 and 4-7 two softmax groups on
// alternating steps, 8 tile loads, 9 issue of S, 10 draws the items and lists the blocks they visit, 11 issue of P V.
// TMEM: S buffer n at columns 128 n (P over its first 64), O at 384.
//
// B=4 S=4096 Hq=32 dense, with the proxy heads: 0.607 ms against 0.767 + 0.492 ms of the key-block stationary kernel and its combine;
// B=1 S=16384 Hq=24 top-k 96 blocks: 1.49 against 2.11 + 1.54 ms.  A step takes 1656 cycles (dense, main heads only, one launch under a
// profiler), of which the tensor core and the special function unit work 1024 each.  It is bound by the way from a finished P through P V,
// S and three hand-offs to the next S in the same buffer, shared by three buffers, and by the softmax of a step beside the other
// group's (about 2000 and 2300 cycles when a step took 1860).  Measured in
// its place, same problem: two heads per CTA with an O and one S buffer each 0.68 ms; the same with two half-block S buffers each
// 0.62; with twice the softmax warps, one set per half block 0.75; one head, a softmax group per half block 0.72; one issuing
// thread for all products 1.00 (it needs 1100 to 2000 cycles for a half block's waits, products and commits).
#include "host_common.h"
#include "launch.h"
#include "msa_common.cuh"
#include "sm100.cuh"
#include "tma_host.h"

namespace fmsa {
namespace {

struct TileParams {
    const uint4* visits;        // [B*Hp][tiles][tiles]: which rows of query tile i selected block j (sparse), or null (dense)
    const int32_t* doc_start;   // [B,S] first token of each token's document (packed sequences), or null
    const float* sinks;         // [Hq] or null
    __nv_bfloat16* out;         // [B,S,Hq*128]
    float* lse;                 // [B,Hq,S]; without the sinks
    float* lse_proxy;           // [B,Hp,S]
    float* zero;                // a scalar to set to zero, or null
    int32_t* counter;
    int32_t* status;
    int32_t n_items;
    int S, B, Hq, Hp, mpp, ppk, pg;
    int tiles;                  // query tiles 0 .. tiles-1 of every (batch, proxy head) are worked on
    int with_proxy;
    float scale_log2e;
};

struct TileItem {
    int32_t i, b, p;
    int32_t h;       // main head inside the proxy head's group; the proxy head itself: mpp
    int32_t steps;   // visited blocks; < 0: no more work
};

constexpr int kTileKvStages = 5, kTileBuffers = 3, kTileRing = 2;
constexpr int kTileThreads = 3 * 128;
// Registers per thread after the warpgroups re-divide the register file: 384 threads are launched with 168.
constexpr int kTileRegsLaunch = 168, kTileRegsSoftmax = 208, kTileRegsMisc = 88;
static_assert(2 * kTileRegsSoftmax + kTileRegsMisc <= 3 * kTileRegsLaunch, "register re-division must balance");
static_assert(kTileRegsLaunch == (65536 / kTileThreads) / 8 * 8, "registers per thread at launch");

struct TileCtrl {
    uint64_t q_full, q_empty, kv_full[kTileKvStages], kv_empty[kTileKvStages];
    uint64_t s_full[kTileBuffers], p_full[kTileBuffers][2], pv_done[kTileBuffers];   // p_full: [half of the keys]
    uint64_t chain[2][4];                        // [group][quarter]
    uint64_t sum_full[2], o_free;                // [group]
    uint64_t item_full[kTileRing], item_empty[kTileRing];
    TileItem items[kTileRing];
    alignas(16) uint4 rows[kTileRing][kTileFwdMaxBlocks];     // per visited block: the rows that selected it
    uint16_t block[kTileRing][kTileFwdMaxBlocks];             // the visited blocks, descending
    float top[128];                                           // running maximum of every row (log2 domain)
    float2 part[2][128];                                      // [group] (max, sum) at the end of an item
    alignas(16) uint32_t off[kTileBuffers][4];                // per S buffer: the rows that did not select the step's block
    uint32_t tmem_slot;
};
constexpr size_t kTileFwdTileBytes = static_cast<size_t>(1 + kTileKvStages) * kTileBytes;
constexpr size_t kTileSmemBytes = kTileFwdTileBytes + 1024 + sizeof(TileCtrl);
static_assert(kTileSmemBytes <= 232448, "shared memory budget of one CTA");

// Rows whose maximum grows by less than this (log2) keep the old one: P is then at most 256 times larger than with the
// new one, the sum is the same, and O need not be rescaled.
constexpr float kLazyRescale = 8.f;
// fp16 P (and with it O and the sum) are 2^7 times larger, at most 2^15, so that the P of a block far below the row's maximum become
// subnormal later.  (The key-block stationary forward takes P relative to the block's own maximum.  One dominant key of value zero in the
// block visited first, S=4096, 12 / 14 / 16 / 18 nats above N(0,1) logits, error of the row against 64 bits: 2.9e-4 / 2.9e-4 / 4.9e-4 /
// 3.2e-3; without the factor 1.0e-3 / 7.5e-3 / 5.7e-2 / 0.38; in the key-block stationary forward 3.9e-4 / 1.4e-3 / 1.0e-2 / 6.6e-2.  That one
// is the better one beyond 22 nats, where such a row of values up to 256 is below fp16's normal numbers itself.  2^11 with a limit of 2^4
// moves this to 25 nats and rescales more often: forward of B=1 S=16384 Hq=24 top-k 96, logits of four times the width, 1.96 -> 2.11 ms.)
template <bool FP16>
constexpr float kLiftP = FP16 ? 7.f : 0.f;

// K and V tiles pass through one ring in the order in which they are needed: K_0 K_1 K_2 V_0 K_3 V_1 .. (proxy head: K_0 K_1 ..).
//   S thread      S of a step, behind the completion of the P V that read P from the same buffer three steps before (products are only
//                 sure to follow one another where accumulator and shape are the same)
//   P V thread    O += P V of a step, in two halves of 64 keys
constexpr uint32_t kHalfRowBytes = 64 * 128;   // rows 64.. of a panel

template <bool FP16, bool VARLEN>
__global__ void __launch_bounds__(kTileThreads, 1) tile_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q,
                                                                   const __grid_constant__ CUtensorMap tmap_k,
                                                                   const __grid_constant__ CUtensorMap tmap_v,
                                                                   const __grid_constant__ CUtensorMap tmap_qp,
                                                                   const __grid_constant__ CUtensorMap tmap_kp, const TileParams P) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t tiles = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t tile_q = tiles, tile_kv = tiles + kTileBytes;
    TileCtrl* sm = reinterpret_cast<TileCtrl*>(smem_raw + (tiles - smem_u32(smem_raw)) + kTileFwdTileBytes);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    auto BAR = [&](uint64_t& b) { return smem_u32(&b); };

    if (tid == 0) {
        mbar_init(BAR(sm->q_full), 1);
        mbar_init(BAR(sm->q_empty), 1);
        mbar_init(BAR(sm->sum_full[0]), 4);
        mbar_init(BAR(sm->sum_full[1]), 4);
        mbar_init(BAR(sm->o_free), 4);
        for (int i = 0; i < 8; ++i) mbar_init(BAR(sm->chain[i >> 2][i & 3]), 1);
        for (int i = 0; i < kTileBuffers; ++i) {
            mbar_init(BAR(sm->s_full[i]), 1);
            mbar_init(BAR(sm->p_full[i][0]), 4);
            mbar_init(BAR(sm->p_full[i][1]), 4);
            mbar_init(BAR(sm->pv_done[i]), 1);
        }
        for (int i = 0; i < kTileKvStages; ++i) {
            mbar_init(BAR(sm->kv_full[i]), 1);
            mbar_init(BAR(sm->kv_empty[i]), 1);
        }
        for (int i = 0; i < kTileRing; ++i) {
            mbar_init(BAR(sm->item_full[i]), 1);
            mbar_init(BAR(sm->item_empty[i]), 11);   // loads, issue (2), eight softmax warps
        }
        fence_mbar_init();
        prefetch_tmap(&tmap_q);
        prefetch_tmap(&tmap_k);
        prefetch_tmap(&tmap_v);
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
    constexpr uint32_t tmem = 0, tmem_o = 128 * kTileBuffers;   // all 512 columns: the allocation starts at column 0
    if (sm->tmem_slot != tmem) {
        wait_for_previous_kernel();   // (a kernel that has left counts as complete for those behind it)
        if (tid == 0) atomicMax(P.status, kStatusBadSmem);
        __syncthreads();
        if (warp == 0) tmem_dealloc(sm->tmem_slot, 512);
        return;
    }

    wait_for_previous_kernel();
    if (P.zero && blockIdx.x == 0 && tid == 0) *P.zero = 0.f;

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
    if (warp >= 8) {
        reg_dec<kTileRegsMisc>();
        if (warp == 10) {
            // =========================== items ===========================
            for (uint32_t draw = 0;; ++draw) {
                const uint32_t slot = draw % kTileRing;
                if (draw >= kTileRing) wait(BAR(sm->item_empty[slot]), (draw / kTileRing - 1) & 1);
                if (bad) break;
                uint32_t u = 0;
                if (lane == 0) u = static_cast<uint32_t>(atomicAdd(P.counter, 1));
                u = __shfl_sync(0xffffffffu, u, 0);
                TileItem it = {};
                it.steps = -1;
                if (u < static_cast<uint32_t>(P.n_items)) {
                    // items of one query tile number: the main heads of every batch element, then its proxy heads
                    const uint32_t mains = P.B * P.Hq, level = mains + (P.with_proxy ? P.B * P.Hp : 0);
                    it.i = P.tiles - 1 - static_cast<int>(u / level);
                    const uint32_t r = u % level;
                    const uint32_t bp = r < mains ? r / P.mpp : r - mains;
                    it.h = r < mains ? r % P.mpp : P.mpp;
                    it.b = static_cast<int>(bp / P.Hp);
                    it.p = static_cast<int>(bp % P.Hp);
                    if (!P.visits) {
                        // dense: every block from the one the first row's document starts in
                        it.steps = it.i + 1;
                        if (VARLEN) it.steps -= min(max(P.doc_start[static_cast<int64_t>(it.b) * P.S + it.i * kBlock] >> 7, 0), it.i);
                    } else {
                        const uint4* src = P.visits + (static_cast<int64_t>(bp) * P.tiles + it.i) * P.tiles;
                        int n = 0;
                        for (int j0 = it.i; j0 >= 0; j0 -= 32) {
                            const int j = j0 - lane;
                            const uint4 w = j >= 0 ? src[j] : make_uint4(0, 0, 0, 0);
                            const bool some = (w.x | w.y | w.z | w.w) != 0;
                            const uint32_t m = __ballot_sync(0xffffffffu, some);
                            const int at = n + __popc(m & ((1u << lane) - 1u));
                            if (some && at < kTileFwdMaxBlocks) {
                                sm->rows[slot][at] = w;
                                sm->block[slot][at] = static_cast<uint16_t>(j);
                            }
                            n += __popc(m);
                        }
                        if (n == 0 && lane == 0) {   // (not from a selection: every row selects its own block)
                            sm->rows[slot][0] = make_uint4(0, 0, 0, 0);
                            sm->block[slot][0] = static_cast<uint16_t>(it.i);
                        }
                        if (n > kTileFwdMaxBlocks) {   // (documents that are longer than the caller said)
                            n = kTileFwdMaxBlocks;
                            if (lane == 0) atomicMax(P.status, kStatusBadIndex);
                        }
                        it.steps = max(n, 1);
                    }
                }
                if (lane == 0) sm->items[slot] = it;
                warp_arrive(BAR(sm->item_full[slot]));
                if (it.steps < 0) break;
            }
        } else if (warp == 8 && elect_one()) {
            // =========================== tile loads ===========================
            uint32_t st = 0, ph = 1, items = 0;   // stage of the ring, phase bit of its kv_empty, items so far
            for (uint32_t draw = 0;; ++draw, ++items) {
                const uint32_t slot = draw % kTileRing;
                wait1(BAR(sm->item_full[slot]), (draw / kTileRing) & 1);
                if (bad) break;
                const TileItem it = sm->items[slot];
                if (it.steps < 0) break;
                const bool px = it.h == P.mpp;
                const int kh = px ? it.p / P.pg : it.p / P.ppk;
                for (int t = -kTileBuffers; t < it.steps && !bad; ++t) {
#pragma unroll 1
                    for (int v = 1; v >= 0; --v) {   // V of step t, K of step t + 3
                        const int k = v ? t : t + kTileBuffers;
                        if (k < 0 || k >= it.steps || (v && px)) continue;
                        wait1(BAR(sm->kv_empty[st]), ph);   // (the first round finds every stage free)
                        if (bad) break;
                        const int j = P.visits ? sm->block[slot][k] : it.i - k;
                        mbar_arrive_expect_tx(BAR(sm->kv_full[st]), kTileBytes);
                        tma_load_tile(tile_kv + st * kTileBytes, v ? &tmap_v : px ? &tmap_kp : &tmap_k, j * kBlock, kh, it.b, BAR(sm->kv_full[st]));
                        if (++st == kTileKvStages) {
                            st = 0;
                            ph ^= 1;
                        }
                    }
                    if (t == -kTileBuffers) {
                        if (items > 0) wait1(BAR(sm->q_empty), (items - 1) & 1);
                        if (bad) break;
                        mbar_arrive_expect_tx(BAR(sm->q_full), kTileBytes);
                        tma_load_tile(tile_q, px ? &tmap_qp : &tmap_q, it.i * kBlock, px ? it.p : it.p * P.mpp + it.h, it.b, BAR(sm->q_full));
                    }
                }
                mbar_arrive(BAR(sm->item_empty[slot]));
            }
        } else if ((warp == 9 || warp == 11) && elect_one()) {
            // =========================== S (warp 9) and P V (warp 11) ===========================
            const bool pv = warp == 11;
            uint32_t st0 = 0, ph0 = 0;       // ring position (stage, phase bit) of the item's first tile
            uint32_t buf = 0, bph = 0;       // S buffer and its phase bit
            for (uint32_t draw = 0;; ++draw) {
                const uint32_t slot = draw % kTileRing;
                wait1(BAR(sm->item_full[slot]), (draw / kTileRing) & 1);
                if (bad) break;
                const int steps = sm->items[slot].steps;
                const bool px = sm->items[slot].h == P.mpp;
                if (steps < 0) break;
                if (!pv) wait1(BAR(sm->q_full), draw & 1);
                // position of K_t: t, and one for every V before it (V_u comes before K_{u + 3}); of V_t: the K up to t + 2 and the V before it
                uint32_t st = st0, ph = ph0;
                auto skip = [&](uint32_t n) {   // n <= kTileKvStages
                    st += n;
                    if (st >= kTileKvStages) {
                        st -= kTileKvStages;
                        ph ^= 1;
                    }
                };
                if (pv) skip(min(steps, kTileBuffers));
#pragma unroll 1
                for (int t = 0; t < steps && !bad; ++t) {
                    const uint32_t at = tile_kv + st * kTileBytes, sbuf = tmem + 128 * buf;
                    if (!pv) {
                        wait1(BAR(sm->kv_full[st]), ph);
                        wait1(BAR(sm->pv_done[buf]), bph ^ 1);   // (the first round finds every buffer free)
                        if (bad) break;
                        tc_fence_after_sync();
                        umma_tile_128<false, false, FP16>(sbuf, tile_q, at, false);   // S = Q K_j^T
                        umma_commit(BAR(sm->s_full[buf]));
                        umma_commit(BAR(sm->kv_empty[st]));
                        skip(t + 1 < kTileBuffers || px ? 1 : 2);
                    } else if (px) {   // nothing to multiply: the buffer is free when it has been read
                        wait1(BAR(sm->p_full[buf][0]), bph);
                        wait1(BAR(sm->p_full[buf][1]), bph);
                        if (bad) break;
                        umma_commit(BAR(sm->pv_done[buf]));
                    } else {
                        wait1(BAR(sm->p_full[buf][0]), bph);
                        wait1(BAR(sm->kv_full[st]), ph);
                        if (bad) break;
                        tc_fence_after_sync();
                        const uint4 off = *reinterpret_cast<const uint4*>(sm->off[buf]);
                        // O += P V_j; where the first block is not every row's, O has been cleared
                        umma_ts_rows<4, 8, FP16>(tmem_o, sbuf, at, t > 0 || (off.x | off.y | off.z | off.w) != 0, off);
                        wait1(BAR(sm->p_full[buf][1]), bph);
                        if (bad) break;
                        tc_fence_after_sync();
                        umma_ts_rows<4, 8, FP16>(tmem_o, sbuf + 32, at + kHalfRowBytes, true, off);
                        umma_commit(BAR(sm->pv_done[buf]));
                        umma_commit(BAR(sm->kv_empty[st]));
                        skip(t + kTileBuffers < steps ? 2 : 1);
                    }
                    if (++buf == kTileBuffers) {
                        buf = 0;
                        bph ^= 1;
                    }
                }
                if (bad) break;
                if (!pv) umma_commit(BAR(sm->q_empty));
                st0 += px ? steps : 2 * steps;
                ph0 ^= st0 / kTileKvStages & 1;
                st0 %= kTileKvStages;
                mbar_arrive(BAR(sm->item_empty[slot]));
            }
        }
    } else {
        reg_inc<kTileRegsSoftmax>();
        // =========================== softmax ===========================
        // Thread = row.  The running maximum of a row is handed from group to group, step by step; either group sums the P of its own
        // steps.  At the end of an item the group that did not have its last step leaves its sum to the other one, which writes the
        // rows while this one is at the next item's first step.
        const int g = warp >> 2;
        const uint32_t chain_in = BAR(sm->chain[g ^ 1][quarter]), chain_out = BAR(sm->chain[g][quarter]);
        const float2 sc2 = make_float2(P.scale_log2e, P.scale_log2e);
        uint32_t step = 0;               // steps so far
        uint32_t buf = 0, bph = 0;       // S buffer and its phase bit
        uint32_t sums = 0;               // phase bits of sum_full
        for (uint32_t draw = 0;; ++draw) {
            const uint32_t slot = draw % kTileRing;
            wait(BAR(sm->item_full[slot]), (draw / kTileRing) & 1);
            if (bad) break;
            const int steps = sm->items[slot].steps, diag = sm->items[slot].i;
            if (steps < 0) break;
            const bool px = sm->items[slot].h == P.mpp;
            const int lo = VARLEN ? P.doc_start[static_cast<int64_t>(sm->items[slot].b) * P.S + diag * kBlock + row] : 0;   // first visible key
            float m = -INFINITY, l = 0.f;   // running maximum (log2 domain), and this group's sum relative to it
            uint32_t last = 0, last_ph = 0; // S buffer of the step before, its phase bit
#pragma unroll 1
            for (int t = 0; t < steps; ++t, ++step) {
                if ((step & 1) == static_cast<uint32_t>(g)) {
                    const uint32_t ts = tmem + 128 * buf;
                    const int j = P.visits ? sm->block[slot][t] : diag - t;
                    // the warp's rows that selected the block
                    const uint32_t word = P.visits ? reinterpret_cast<const uint32_t*>(&sm->rows[slot][t])[quarter]
                                                   : (VARLEN ? __ballot_sync(0xffffffffu, (lo >> 7) <= j) : 0xffffffffu);
                    const bool sel = word >> lane & 1;
                    bool clear = false;   // the first block is not every row's (not from a selection): such rows start from zeros
                    if (P.visits && t == 0 && !px) {
                        const uint4 w = sm->rows[slot][0];
                        clear = (w.x & w.y & w.z & w.w) != 0xffffffffu;
                    }
                    const int lowc = VARLEN && (lo >> 7) == j ? lo & 127 : 0;   // first visible key inside the block
                    wait(BAR(sm->s_full[buf]), bph);
                    if (bad) break;
                    tc_fence_after_sync();
                    if (lane == 0) sm->off[buf][quarter] = ~word;   // (the product that read the buffer's last ones has completed)
                    if (j == diag || (VARLEN && __any_sync(0xffffffffu, lowc > 0))) {   // the causal edge, or the start of the row's document:
                        const int limit = j == diag ? row : 127;                        // hidden logits become -inf
#pragma unroll 1
                        for (int c = 0; c < 128; c += 16) {
                            uint32_t v[16];
                            tmem_ld16(tmem_addr(ts, quarter, c), v);
                            tmem_ld_wait();
#pragma unroll
                            for (int y = 0; y < 16; ++y)
                                if (c + y > limit || (VARLEN && c + y < lowc)) v[y] = 0xff800000u;
                            tmem_st16(tmem_addr(ts, quarter, c), v);
                        }
                        tmem_st_wait();
                    }
                    uint32_t s[4][32];
                    float mx0 = -INFINITY, mx1 = -INFINITY;
                    tmem_ld32(tmem_addr(ts, quarter, 0), s[0]);
                    tmem_ld32(tmem_addr(ts, quarter, 32), s[1]);
                    tmem_ld_wait();
                    tmem_ld32(tmem_addr(ts, quarter, 64), s[2]);
                    tmem_ld32(tmem_addr(ts, quarter, 96), s[3]);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (c == 2) tmem_ld_wait();
#pragma unroll
                        for (int y = 0; y < 32; y += 4) {
                            mx0 = fmax3(mx0, __uint_as_float(s[c][y]), __uint_as_float(s[c][y + 1]));
                            mx1 = fmax3(mx1, __uint_as_float(s[c][y + 2]), __uint_as_float(s[c][y + 3]));
                        }
                    }
                    const float mt = fmaxf(mx0, mx1) * P.scale_log2e;   // raw logits: scale > 0, so the maximum commutes with it
                    if (step) wait(chain_in, g ? (step >> 1) & 1 : ((step >> 1) - 1) & 1);
                    if (bad) break;
                    const float top = t > 0 ? sm->top[row] : -INFINITY;   // the row's maximum so far
                    const bool any_raise = __any_sync(0xffffffffu, sel && mt > top + kLazyRescale);
                    const float mn = any_raise && sel ? fmaxf(top, mt) : top;
                    if (any_raise || t == 0) sm->top[row] = mn;
                    warp_arrive(chain_out);
                    if (mn != m) {   // (raised here or by the other group)
                        l *= m == -INFINITY ? 0.f : fast_exp2(m - mn);
                        m = mn;
                    }
                    if (!px && any_raise && t > 0) {
                        // the product of the step before may still be adding to O
                        wait(BAR(sm->pv_done[last]), last_ph);
                        if (bad) break;
                        tc_fence_after_sync();
                        const float alpha = top == -INFINITY ? 0.f : fast_exp2(top - mn);
                        const float2 a2 = make_float2(alpha, alpha);
#pragma unroll 1
                        for (int c = 0; c < 128; c += 16) {
                            uint32_t o[16];
                            tmem_ld16(tmem_addr(tmem_o, quarter, c), o);
                            tmem_ld_wait();
#pragma unroll
                            for (int y = 0; y < 16; y += 2) {
                                const float2 r = f2_mul(f2_from_bits(o[y], o[y + 1]), a2);
                                o[y] = __float_as_uint(r.x);
                                o[y + 1] = __float_as_uint(r.y);
                            }
                            tmem_st16(tmem_addr(tmem_o, quarter, c), o);
                        }
                    }
                    const float nm = m == -INFINITY ? 0.f : kLiftP<FP16> - m;   // (a row that has not selected anything yet)
                    const float2 nm2 = make_float2(nm, nm);
                    float2 l2a = make_float2(0.f, 0.f), l2b = make_float2(0.f, 0.f);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        uint32_t pk[16];
#pragma unroll
                        for (int y = 0; y < 32; y += 4) {
                            const float2 a = f2_fma(f2_from_bits(s[c][y], s[c][y + 1]), sc2, nm2);
                            const float2 b = f2_fma(f2_from_bits(s[c][y + 2], s[c][y + 3]), sc2, nm2);
                            const float2 pa = make_float2(fast_exp2(a.x), fast_exp2(a.y)), pb = make_float2(fast_exp2(b.x), fast_exp2(b.y));
                            l2a = f2_add(l2a, pa);
                            l2b = f2_add(l2b, pb);
                            pk[y >> 1] = pack_act<FP16>(pa.x, pa.y);
                            pk[(y >> 1) + 1] = pack_act<FP16>(pb.x, pb.y);
                        }
                        if (!px) tmem_st16(tmem_addr(ts, quarter, 16 * c), pk);
                        if (c & 1) {
                            // the first product of an item overwrites O: the rows of the item before must have been read
                            if (c == 1 && t == 0) {
                                if (draw > 0) wait(BAR(sm->o_free), (draw - 1) & 1);
                                if (clear) {
                                    tc_fence_after_sync();
                                    const uint32_t zero[16] = {};
#pragma unroll 1
                                    for (int o = 0; o < 128; o += 16) tmem_st16(tmem_addr(tmem_o, quarter, o), zero);
                                }
                            }
                            if (!px) tmem_st_wait();
                            tc_fence_before_sync();
                            warp_arrive(BAR(sm->p_full[buf][c >> 1]));
                        }
                    }
                    if (sel) l += (l2a.x + l2a.y) + (l2b.x + l2b.y);
                }
                last = buf;
                last_ph = bph;
                if (++buf == kTileBuffers) {
                    buf = 0;
                    bph ^= 1;
                }
            }
            if (bad) break;
            // ---- the end of the item
            const int other = step & 1;   // the group that did not have the last step
            if (g == other) {
                sm->part[g][row] = make_float2(m, l);
                warp_arrive(BAR(sm->sum_full[g]));
                warp_arrive(BAR(sm->item_empty[slot]));
            } else {
                const TileItem it = sm->items[slot];
                const int q = it.i * kBlock + row;
                wait(BAR(sm->sum_full[other]), (sums >> other) & 1);
                if (bad) break;
                const float2 a = sm->part[other][row];
                // (maxima only rise: this group's is the latest)
                l += a.x == -INFINITY ? 0.f : a.y * fast_exp2(a.x - m);
                const float lse = l > 0.f ? (m + (__log2f(l) - kLiftP<FP16>)) * kLn2 : (l == 0.f ? -INFINITY : l);   // (a NaN stays one)
                if (px) {
                    P.lse_proxy[(static_cast<int64_t>(it.b) * P.Hp + it.p) * P.S + q] = lse;
                } else {
                    const int head = it.p * P.mpp + it.h;
                    P.lse[(static_cast<int64_t>(it.b) * P.Hq + head) * P.S + q] = lse;
                    if (P.sinks) l += fast_exp2(P.sinks[head] * kLog2e + (m == -INFINITY ? 0.f : kLiftP<FP16> - m));
                    const float inv = l == 0.f ? 0.f : 1.f / l;
                    const float2 inv2 = make_float2(inv, inv);
                    wait(BAR(sm->pv_done[last]), last_ph);
                    if (bad) break;
                    tc_fence_after_sync();
                    __nv_bfloat16* to = P.out + (static_cast<int64_t>(it.b) * P.S + q) * (static_cast<int64_t>(P.Hq) * kHeadDim) +
                                        static_cast<int64_t>(head) * kHeadDim;
#pragma unroll 1
                    for (int c = 0; c < 128; c += 64) {
                        uint32_t o[2][32];
                        tmem_ld32(tmem_addr(tmem_o, quarter, c), o[0]);
                        tmem_ld32(tmem_addr(tmem_o, quarter, c + 32), o[1]);
                        tmem_ld_wait();
                        if (c == 64) {
                            tc_fence_before_sync();
                            warp_arrive(BAR(sm->o_free));
                        }
#pragma unroll
                        for (int y = 0; y < 64; y += 8) {
                            uint32_t pk[4];
#pragma unroll
                            for (int z = 0; z < 8; z += 2) {
                                const float2 r = f2_mul(f2_from_bits(o[y >> 5][(y & 31) + z], o[y >> 5][(y & 31) + z + 1]), inv2);
                                pk[z >> 1] = pack_act<FP16>(r.x, r.y);
                            }
                            *reinterpret_cast<uint4*>(to + c + y) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                        }
                    }
                }
                if (px) warp_arrive(BAR(sm->o_free));
                warp_arrive(BAR(sm->item_empty[slot]));
            }
            sums ^= 1u << other;
        }
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

// The sinks join the log-sum-exps behind the kernel above (which has used them for `out`): lse = log(exp(lse) + exp(sink)).  The KL
// teacher's rows then sum to T = mean_h exp(lse_h - lse'_h), and the proxy log-sum-exp is lowered by log T (see combine_lse_kernel).
// One thread per (batch, proxy head, query position).
__global__ void __launch_bounds__(256) sink_lse_kernel(float* __restrict__ lse, float* __restrict__ lse_proxy, const float* __restrict__ sinks,
                                                       int B, int Hp, int mpp, int S, int rows) {
    wait_for_previous_kernel();
    const int64_t t = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
    if (t >= static_cast<int64_t>(B) * Hp * rows) return;
    const int q = static_cast<int>(t % rows);
    const int64_t bp = t / rows;
    const int p = static_cast<int>(bp % Hp);
    float keep = 0.f;
    for (int h = 0; h < mpp; ++h) {
        float* at = lse + (bp * mpp + h) * S + q;
        const float raw = *at, sk = sinks[p * mpp + h];
        const float with = fmaxf(raw, sk) + log1pf(expf(-fabsf(raw - sk)));
        keep += expf(raw - with);
        *at = with;
    }
    if (lse_proxy) lse_proxy[bp * S + q] -= logf(keep / static_cast<float>(mpp));
}

}  // namespace

int launch_tile_fwd(const fmsa_problem* pb, const fmsa_tensor* q, const fmsa_tensor* k, const fmsa_tensor* v, const fmsa_tensor* q_proxy,
                    const fmsa_tensor* k_proxy, const void* visits, void* out, float* lse, float* lse_proxy, const float* sinks, float* zero,
                    int tiles, int dense, int32_t* counter, int32_t* status, cudaStream_t st) {
    FMSA_REQUIRE(problem_ok(pb) && q && k && v && q->ptr && k->ptr && v->ptr && out && lse && counter && status);
    FMSA_REQUIRE(dense || visits);
    FMSA_REQUIRE(!lse_proxy || (q_proxy && k_proxy && q_proxy->ptr && k_proxy->ptr));
    FMSA_REQUIRE(tiles >= 1 && tiles <= pb->S / kBlock && (dense || tiles <= kTileFwdMaxTiles) && pb->scale > 0.f);
    FMSA_REQUIRE(aligned16(out) && (reinterpret_cast<uintptr_t>(visits) & 15u) == 0);
    const fmsa_tensor* qp = lse_proxy ? q_proxy : q;
    const fmsa_tensor* kp = lse_proxy ? k_proxy : k;
    for (const fmsa_tensor* t : {q, k, v, qp, kp}) FMSA_REQUIRE(tma_compatible(t->ptr, t->stride_b, t->stride_h, t->stride_s));
    CUtensorMap tq, tk, tv, tqp, tkp;
    auto map = [&](CUtensorMap* m, const fmsa_tensor* t, int heads) {
        return make_tmap_bhsd(m, t->ptr, pb->B, heads, pb->S, t->stride_b, t->stride_h, t->stride_s, 128);
    };
    if (!map(&tq, q, pb->Hq) || !map(&tk, k, pb->Hkv) || !map(&tv, v, pb->Hkv) || !map(&tqp, qp, lse_proxy ? pb->Hp : pb->Hq) ||
        !map(&tkp, kp, lse_proxy ? pb->Hpkv : pb->Hkv))
        return FMSA_ERR_CUDA;
    TileParams P;
    P.visits = dense ? nullptr : static_cast<const uint4*>(visits);
    P.doc_start = pb->doc_start; P.sinks = sinks;
    P.out = static_cast<__nv_bfloat16*>(out); P.lse = lse; P.lse_proxy = lse_proxy; P.zero = zero;
    P.counter = counter; P.status = status;
    P.S = pb->S; P.B = pb->B; P.Hq = pb->Hq; P.Hp = pb->Hp;
    P.mpp = pb->Hq / pb->Hp; P.ppk = pb->Hp / pb->Hkv; P.pg = pb->Hp / pb->Hpkv;
    P.tiles = tiles; P.with_proxy = lse_proxy ? 1 : 0; P.scale_log2e = pb->scale * kLog2e;
    const int sms = device_sm_count();
    const int64_t bps = static_cast<int64_t>(pb->B) * pb->Hp;
    const int64_t items = tiles * (static_cast<int64_t>(pb->B) * pb->Hq + (P.with_proxy ? bps : 0));
    FMSA_REQUIRE(items < 0x7f000000LL);   // (the work counter runs past the end by one per CTA)
    P.n_items = static_cast<int32_t>(items);
    const bool fp16 = pb->dtype == FMSA_DTYPE_FP16, varlen = pb->doc_start != nullptr;
    using KernelFn = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, TileParams);
    static const KernelFn kernels[4] = {tile_fwd_kernel<false, false>, tile_fwd_kernel<false, true>, tile_fwd_kernel<true, false>,
                                        tile_fwd_kernel<true, true>};
    const KernelFn kernel = kernels[(fp16 ? 2 : 0) + (varlen ? 1 : 0)];
    if (sms <= 0 || !ensure_smem_attr(reinterpret_cast<const void*>(kernel), kTileSmemBytes)) return FMSA_ERR_CUDA;
    const int grid = P.n_items < sms ? P.n_items : sms;
    launch_chained(kernel, grid, kTileThreads, kTileSmemBytes, st, tq, tk, tv, tqp, tkp, P);
    if (sinks) {
        const int64_t threads = bps * tiles * kBlock;
        launch_chained(sink_lse_kernel, static_cast<unsigned>((threads + 255) / 256), 256, 0, st, lse, lse_proxy, sinks, pb->B, pb->Hp, P.mpp, pb->S, tiles * kBlock);
    }
    return check_launch();
}

}  // namespace fmsa

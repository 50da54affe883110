// Index arithmetic shared by the forward, combine and backward kernels.
#pragma once

#include <stdint.h>

#include "sm100.cuh"

namespace fmsa {

// Dense (warmup) schedule: the "reverse-index row" of key block j of one (batch, proxy head) is
// every query position >= 128*j, in order.  Rows are laid out back to back, so the edge of
// (key block j, query q) sits at  bp*S*(NB+1)/2 + j*S - 128*j*(j-1)/2 + (q - 128*j).
__host__ __device__ __forceinline__ int64_t dense_edges_per_bp(int S, int NB) {
    return static_cast<int64_t>(S) * (NB + 1) / 2;
}
__host__ __device__ __forceinline__ int64_t dense_edge_base(int64_t bp, int S, int NB) {
    return bp * dense_edges_per_bp(S, NB);
}
__host__ __device__ __forceinline__ int64_t dense_row_offset(int j, int S) {
    return static_cast<int64_t>(j) * S - static_cast<int64_t>(kBlock) * j * (j - 1) / 2;
}

// -------------------------------------------------------------------------------------------
// Work decomposition shared by the forward and the backward.
//
// A reverse-index row (batch, proxy head, key block j) can hold anything from one chunk of 128
// query rows to all S - 128*j later rows (a "sink" block).  To keep the persistent CTAs balanced a
// row is cut into sub-units of at most C chunks (chunks_per_subunit below).  The number of rows is only known
// on the device, so the sub-units are enumerated for the worst case (NB - j chunks) and a CTA that
// draws a sub-unit beyond the real end of its row simply skips it.
//
// Order: (batch, KV head) group major, then sub-unit index s (chunks C*s .. C*s+C-1 of a row), then key
// block ascending, then proxy head of the group.  Group-major order keeps the rows that the active
// CTAs gather from and reduce into (a few heads of Q, dO) resident in L2.  Inside a group, putting s
// outermost makes neighbouring sub-units alike in size (for a given s the rows of neighbouring key
// blocks are about equally long, and the sub-units that lie beyond the end of their row cluster
// together), so both a dynamic work counter and a static round-robin deal stay balanced.
// -------------------------------------------------------------------------------------------
constexpr int kMaxChunksPerSubUnit = 16;

// Key blocks j that can have a sub-unit s: NB - j > C*s, i.e. j < NB - C*s.
// (`depth`: most chunks a row can have; NB, or NB - T where the rows hold query positions of tiles T, T+1, .. only.)
__host__ __device__ __forceinline__ int64_t subunits_per_group(int NB, int depth, int ppk, int C) {
    // sum over s = 0 .. n-1 of (NB - C*s), n = ceil(depth / C)
    const int64_t n = (depth + C - 1) / C;
    return (n * NB - C * (n * (n - 1) / 2)) * ppk;
}

// C for a launch: the largest power of two up to 8 that still leaves every CTA `kSubUnitsPerCta` sub-units on average, or 16
// where that leaves it `kLongSubUnitsPerCta`.  A sub-unit loads K and V once and flushes dV and dK once, so long ones save
// traffic; short ones fill the SMs and bound the tail of the launch: a problem of a few dozen chunks otherwise runs on a
// handful of SMs (B=1, S=1024, Hq=8, top-k 4 blocks: 64 chunks on 16 CTAs).
// The averages are those of an upper bound: `edges` is what the host knows without a look at the selection, S * top_k_blocks
// per proxy head in the sparse schedule.  Early rows have fewer blocks to select, and documents hide some: 77 % of it are
// there at S=4096 top-k 16 blocks, 63 % at S=16384 top-k 96, 48 % with five documents at S=8192 top-k 16, so a launch can
// have half the sub-units per CTA that the constants say.  Both constants were measured with this bound (and the lengths below
// chosen by it).  A row of the reverse index is on average half a chunk longer than its edges.  Where most
// sub-units lie beyond the end of their rows (they are passed over 32 at a time, or to the next one with work: draw_work), C does
// not go below what keeps the enumeration at `kDrawsPerCta` per CTA: shorter ones gain nothing there and flush dV and dK more often.
// Backward kernels with a limit of 16 / 32 / 64 / none: B=4 S=3968 Hq=16 top-k 2 blocks 210 / 209 / 246 / 247 us, B=1 S=52736 Hq=12 top-k 2 with six
// documents 578 / 578 / 601 / 625, B=1 S=41216 Hq=32 top-k 3 and S=65536 Hq=8 top-k 32 equal within the spread of 3 %.
// With 16 the rows of a group are gathered in half as many sweeps, which counts where they do not fit L2 (B=1 S=65536 Hq=8
// top-k 32 blocks, 14 sub-units per CTA: forward 1.70 -> 1.56 ms, backward 3.83 -> 3.49 ms), and K, V, dK and dV move half as often
// (B=2 S=8192 Hq=32 top-k 16 blocks, 7 per CTA, with the last groups cut finer: backward kernels 1.569 -> 1.516 ms; at two per CTA no
// better, with four sub-units of 8 as the least elsewhere B=1 S=16384 top-k 96: 5.58 -> 6.18 ms).
constexpr int kTailFreeGroup = 2;   // (see enumerate_subunits)
constexpr int kSubUnitsPerCta = 6, kLongSubUnitsPerCta = 4, kDrawsPerCta = 32;
inline int chunks_per_subunit(int64_t edges, int64_t groups, int NB, int depth, int ppk, int sms) {
    const int64_t chunks = (edges + kBlock - 1) / kBlock + groups * ppk * NB / 2;
    int c = chunks >= static_cast<int64_t>(kMaxChunksPerSubUnit) * kLongSubUnitsPerCta * sms ? kMaxChunksPerSubUnit : kMaxChunksPerSubUnit / 2;
    while (c > 1 && chunks < static_cast<int64_t>(c) * kSubUnitsPerCta * sms &&
           groups * subunits_per_group(NB, depth, ppk, c / 2) <= static_cast<int64_t>(kDrawsPerCta) * sms)
        c >>= 1;
    return c;
}

// -------------------------------------------------------------------------------------------
// Which query tiles the query-tile stationary forward (tile_fwd.cu) takes: the first `forward_tiles` ones.
// -------------------------------------------------------------------------------------------
constexpr int kTileFwdMaxBlocks = 256;   // most blocks that a tile of a sparse call can visit there
// Query tile i visits up to i + 1 blocks there, against min(i + 1, top_k_blocks) edges per row here, and an edge of the key-block
// stationary forward and its combine takes as long as about two visits: 18.8 ns against 9.0 ns of the whole GPU per 128 edges, or visit,
// of a main head (B=2 S=8192 Hq=32 top-k 16 blocks; B=4 S=4096 Hq=32 dense, both with the proxy heads), and its scattered rows cost more
// power, which is what limits the clock.  So the first 2.5 top_k_blocks tiles go there (forward of B=2 S=8192 Hq=32 top-k 16, back to back:
// 2.0 1127, 2.5 1118, 3.0 1164 us; of B=1 S=32768 top-k 64 12.20, 12.10, 12.30 ms); all of them, so that the other forward and its
// combine need not run, where those would be short (their launches and tails cost as much as some 2800 visits), and where documents are
// known to be so short that no tile sees more than that many blocks (`visible`, 0: not known; B=1 S=8192 Hq=32 top-k 16 as five documents:
// forward 0.333 -> 0.189 ms).  The lists of visited blocks are kept for kTileFwdMaxBlocks, the bit maps behind them for sequences of kTileFwdMaxTiles.
constexpr int kTileFwdLaunchVisits = 2800, kTileFwdMaxTiles = 512;
inline int forward_tiles(int NB, int top_k_blocks, int64_t main_heads, int dense, int visible) {   // main_heads: of all batch elements
    if (dense) return NB;
    int t = 5 * top_k_blocks / 2;
    if (visible > 0 && visible <= t && visible <= kTileFwdMaxBlocks && NB <= kTileFwdMaxTiles) return NB;
    if (NB <= kTileFwdMaxBlocks) {
        if (t >= NB) return NB;
        const int64_t visits = (static_cast<int64_t>(NB) * (NB + 1) - static_cast<int64_t>(t) * (t + 1)) / 2;   // of the tiles from t on
        const int64_t edges = static_cast<int64_t>(NB - t) * top_k_blocks;
        if ((visits - 2 * edges) * main_heads <= kTileFwdLaunchVisits) return NB;
    }
    return t < kTileFwdMaxBlocks ? t : kTileFwdMaxBlocks;
}

// The sub-units of a launch.  Those of the last groups are cut finer (a quarter of the chunks): a group of B=2 S=8192 Hq=32 top-k 16
// blocks has fewer sub-units than there are SMs, so that the launch ended with SMs waiting for one last long sub-unit each: they were
// busy 95-96 % of the kernels' time, 92 % at B=4 S=4096 Hq=16, 79-85 % with five documents at S=8192.  With the long sub-units above and
// finer last groups, backward kernels: 1.550 -> 1.516, 0.694 -> 0.677, 0.522 -> 0.487 ms; halves instead of quarters: 0.499 with the
// documents.
struct SubUnits {
    int32_t n;                                  // all of them (an upper bound of those with work)
    uint32_t n_bulk, per_group, per_group_tail; // indices below n_bulk: per_group for each of the first groups; then per_group_tail each
    int32_t groups_bulk, NB, ppk, chunks, chunks_tail;
};
// False: more sub-units than the work counter can hold (it may run past the end by one per CTA and 31).
inline bool enumerate_subunits(SubUnits* U, int64_t edges, int64_t groups, int NB, int depth, int ppk, int sms) {
    U->NB = NB;
    U->ppk = ppk;
    U->chunks = chunks_per_subunit(edges, groups, NB, depth, ppk, sms);
    U->chunks_tail = U->chunks >= 4 ? U->chunks / 4 : 1;
    // Enough groups that the CTAs have about half a sub-unit's worth of work each left when the finer ones begin (a whole one: 0.705 ms at
    // S=4096, 0.521 with the documents).  A group of several times as much work ends in enough sub-units of its own, the ends of its
    // rows (B=1 S=65536 top-k 32: SMs 99.8 % busy).
    const int64_t tail = static_cast<int64_t>(U->chunks) * sms / 2, per = (edges / groups + kBlock - 1) / kBlock + 1;
    int64_t fine = per > kTailFreeGroup * tail || U->chunks == 1 ? 0 : (tail + per - 1) / per;
    if (fine > groups) fine = groups;
    constexpr int64_t kMost = 0x7f000000LL;
    if (subunits_per_group(NB, depth, ppk, U->chunks_tail) * groups >= kMost) fine = 0;
    // (As above, they stay coarser where there would be too many to draw: B=4 S=3968 Hq=16 top-k 2 blocks 735 -> 717 us, B=1 S=41216 Hq=32
    // top-k 3 2993 -> 2907.  A limit of 64 per CTA has the former at 754 and the latter as it is.)
    while (fine > 0 && subunits_per_group(NB, depth, ppk, U->chunks) * (groups - fine) + subunits_per_group(NB, depth, ppk, U->chunks_tail) * fine >
                           static_cast<int64_t>(kDrawsPerCta) * sms) {
        U->chunks_tail *= 2;
        if (U->chunks_tail >= U->chunks) fine = 0;
    }
    U->groups_bulk = static_cast<int32_t>(groups - fine);
    const int64_t pg = subunits_per_group(NB, depth, ppk, U->chunks), pt = subunits_per_group(NB, depth, ppk, U->chunks_tail);
    if (pg * (groups - fine) + pt * fine >= kMost) return false;
    U->per_group = static_cast<uint32_t>(pg);
    U->per_group_tail = static_cast<uint32_t>(pt);
    U->n_bulk = static_cast<uint32_t>(pg * (groups - fine));
    U->n = static_cast<int32_t>(U->n_bulk + pt * fine);
    return true;
}

struct SubUnit {
    int g, j, pp, chunk0, chunks;
};
// (32-bit arithmetic: 64-bit divisions cost kilobytes of code here.)
__device__ __forceinline__ SubUnit decode_subunit(uint32_t u, const SubUnits& U) {
    SubUnit su;
    const bool bulk = u < U.n_bulk;
    const uint32_t per_group = bulk ? U.per_group : U.per_group_tail;
    su.chunks = bulk ? U.chunks : U.chunks_tail;
    if (!bulk) u -= U.n_bulk;
    su.g = static_cast<int>(u / per_group);
    const uint32_t r = u - su.g * per_group, ppk = U.ppk;
    if (!bulk) su.g += U.groups_bulk;
    su.pp = static_cast<int>(r % ppk);
    int x = static_cast<int>(r / ppk);
    int left = U.NB, s = 0;   // key blocks that have a sub-unit s
    while (x >= left) {   // at most NB / chunks iterations
        x -= left;
        left -= su.chunks;
        s += su.chunks;
    }
    su.j = x;
    su.chunk0 = s;
    return su;
}

// The first sub-unit from `u` on that has work if it lies in u's group, else the first one of the next group; a warp's job, and every lane
// gets the result.  One look at the lengths of the rows finds it: a row can have work in u's sweep, at a place not before u's, or else in the
// next one (work in a later sweep means work in this one too).
template <class RowLength>
__device__ __forceinline__ uint32_t next_subunit(uint32_t u, const SubUnits& U, int g_begin, RowLength&& row_length) {
    const SubUnit su = decode_subunit(u, U);
    const uint32_t lane = threadIdx.x & 31, ppk = U.ppk, g = g_begin + su.g;
    const uint32_t here = su.j * ppk + su.pp, rows = (U.NB - su.chunk0) * ppk;   // u's place in its sweep, and the sweep's size
    const uint32_t group_end = u < U.n_bulk ? (su.g + 1) * U.per_group : U.n_bulk + (su.g + 1 - U.groups_bulk) * U.per_group_tail;
    uint32_t best = group_end - (u - here);   // from the beginning of u's sweep
#pragma unroll 4
    for (uint32_t i = lane; i < rows; i += 32) {
        const uint32_t j = i / ppk;
        const int chunks = (row_length((g * ppk + (i - j * ppk)) * U.NB + j) + kBlock - 1) / kBlock;
        if (chunks > su.chunk0 && i >= here) best = min(best, i);
        else if (chunks > su.chunk0 + su.chunks) best = min(best, rows + i);
    }
    return u - here + __reduce_min_sync(0xffffffffu, best);
}

// What a launch needs to enumerate its sub-units; a member of the parameters of the backward kernels.
struct UnitSpace {
    const int32_t* row_ptr;
    int32_t* counter;
    SubUnits sub;
    int S, NB, Hkv, Hp, ppk, g_begin, dense;
};

// A sub-unit as the drawing thread publishes it to the other roles (kept small: it shares the last 3 KB of shared memory).
struct UnitRec {
    int64_t e0;                      // position of the reverse-index row in col_q / the slot space
    int32_t n;                       // its length
    uint16_t j, b, kvh, p, chunk0;   // (B*Hp < 65536 and S/128 <= 2048 are required by the entry points)
    int16_t chunk1;                  // < 0: no more work
};

// One warp draws the next sub-unit with work (false: none left); `load(u)` fetches sub-unit u and says whether it has any, and
// lane 0 keeps what it fetched.  When the drawn one lies beyond the end of its row the lanes have looked at the 31 behind
// it as well, and the counter moves past those of them that are empty too.  (With a draw for each empty one, about half of
// them at B=2 S=8192 Hq=32 top-k 16 blocks: forward 0.674 -> 0.669 ms, backward kernels 1.539 -> 1.527 ms.)
// Where all 32 are empty it moves on to `next(u)`: the windows of the CTAs overlap, so with a few blocks selected from a long sequence
// they spent most of the time on passing over empty sub-units, each round for a few dozen (B=1 S=52736 Hq=12 top-k 2 blocks, six
// documents: forward 816 -> 247 us, backward kernels 1585 -> 433; B=1 S=65536 Hq=8 top-k 32: 1605 -> 1560, 3445 -> 3388).
template <class Load, class Next>
__device__ __forceinline__ bool draw_work(int32_t* counter, uint32_t n_subunits, Load&& load, Next&& next) {
    const uint32_t lane = threadIdx.x & 31;
    for (;;) {
        uint32_t u = 0;
        if (lane == 0) u = static_cast<uint32_t>(atomicAdd(counter, 1));
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= n_subunits) return false;
        const bool has = u + lane < n_subunits && load(u + lane);
        const uint32_t work = __ballot_sync(0xffffffffu, has);
        if (work & 1u) return true;
        const uint32_t to = work ? u + __ffs(work) - 1 : max(u + 32, next(u));
        if (lane == 0) atomicMax(counter, static_cast<int32_t>(to));
    }
}

// A warp draws and decodes the next sub-unit; the result is lane 0's.
__device__ __forceinline__ UnitRec draw_subunit(const UnitSpace& U) {
    UnitRec nu;
    const bool more = draw_work(U.counter, static_cast<uint32_t>(U.sub.n), [&](uint32_t u) -> bool {
        const SubUnit su = decode_subunit(u, U.sub);
        const uint32_t g = U.g_begin + su.g;
        const int b = g / static_cast<uint32_t>(U.Hkv), kvh = g % static_cast<uint32_t>(U.Hkv), p = kvh * U.ppk + su.pp;
        const int64_t bp = static_cast<int64_t>(b) * U.Hp + p;
        int64_t e0;
        int n;
        if (U.dense) {
            e0 = dense_edge_base(bp, U.S, U.NB) + dense_row_offset(su.j, U.S);
            n = U.S - su.j * kBlock;
        } else {
            e0 = U.row_ptr[bp * U.NB + su.j];
            n = U.row_ptr[bp * U.NB + su.j + 1] - static_cast<int>(e0);
        }
        nu.j = static_cast<uint16_t>(su.j); nu.b = static_cast<uint16_t>(b); nu.kvh = static_cast<uint16_t>(kvh);
        nu.p = static_cast<uint16_t>(p); nu.n = n; nu.e0 = e0;
        nu.chunk0 = static_cast<uint16_t>(su.chunk0);
        nu.chunk1 = static_cast<int16_t>(min((n + kBlock - 1) / kBlock, su.chunk0 + su.chunks));
        return su.chunk0 * kBlock < n;
    }, [&](uint32_t u) -> uint32_t {
        return next_subunit(u, U.sub, U.g_begin, [&](uint32_t row) { return U.row_ptr[row + 1] - U.row_ptr[row]; });
    });
    if (!more) nu.chunk1 = -1;
    return nu;
}
// CSR position of the first slot of a pass over the groups from g_begin on.
__device__ __forceinline__ int64_t first_slot(const UnitSpace& U) {
    return U.dense ? dense_edge_base(static_cast<int64_t>(U.g_begin) * U.ppk, U.S, U.NB)
                   : static_cast<int64_t>(U.row_ptr[static_cast<int64_t>(U.g_begin) * U.ppk * U.NB]);
}

}  // namespace fmsa

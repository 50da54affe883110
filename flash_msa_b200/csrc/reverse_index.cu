// Deterministic reverse index: a CSR that lists, for every (batch, proxy head, key block), the
// query positions that selected that block, in ascending order.
//
// Small kernels, no global atomics and no host synchronisation:
//   1. count : one CTA per (batch*proxy head, query block) builds a shared-memory bitmap
//              "row r selected key block j" and writes the per-(query block, key block) counts
//              (as a stage; in a whole pass the fused selection leaves them);
//   2. colscan: one thread per (batch*proxy head, key block) turns the counts of its column into
//              exclusive offsets over the query blocks and records the column total;
//   3. rowscan: a single CTA turns the totals into row_ptr
//              (2 and 3 are one kernel where that is enough: one_scan);
//   4. fill  : the bitmap is rebuilt and every edge gets position
//              row_ptr + block offset + (number of lower rows of its block that chose the key block).
// The edge rule `0 <= kb < NB && kb <= q/128` is the reference's
// (flash_msa/csrc/reverse_index_cuda.cu:41); its atomics-based slot assignment (:118) is replaced
// by ranks, so the output is a pure function of the input.
#include <mutex>

#include "host_common.h"
#include "launch.h"
#include "sm100.cuh"

namespace fmsa {
namespace {

// Shared memory of the count and fill kernels: the bitmap words[j*4 + w] (rows 32w..32w+31 of the query block that
// selected key block j), then the query block's 128 x Kb selections, copied in with 16-byte loads (the rows of a
// query block are contiguous).  Thread r works on row r and walks its Kb slots starting at slot r % Kb, so that the
// lanes of a warp touch different banks.
__device__ __forceinline__ int32_t* stage_rows(uint32_t* words, const int32_t* idx_rows, int NB, int Kb) {
    int32_t* tile = reinterpret_cast<int32_t*>(words + NB * 4);
    const int4* src = reinterpret_cast<const int4*>(idx_rows);
    int4* dst = reinterpret_cast<int4*>(tile);
    for (int t = threadIdx.x; t < kBlock * Kb / 4; t += blockDim.x) dst[t] = src[t];
    for (int t = threadIdx.x; t < NB * 4; t += blockDim.x) words[t] = 0u;
    __syncthreads();
    return tile;
}
__device__ __forceinline__ int rotated_slot(int s, int r, int Kb) {
    const int x = s + (r % Kb);
    return x >= Kb ? x - Kb : x;
}
__device__ __forceinline__ void build_bitmap(uint32_t* words, const int32_t* tile, int NB, int Kb, int qblk) {
    const int r = threadIdx.x;   // 128 threads: one per row
    const int32_t* row = tile + r * Kb;
    for (int s = 0; s < Kb; ++s) {
        const int j = row[rotated_slot(s, r, Kb)];
        if (static_cast<unsigned>(j) < static_cast<unsigned>(NB) && j <= qblk) atomicOr(&words[j * 4 + (r >> 5)], 1u << (r & 31));
    }
    __syncthreads();
}

// With `visits` the bitmaps of query tiles below `tiles` also go to memory: tile_fwd.cu walks the blocks in them.  `counts` null:
// nothing else (the grid then has those query tiles only).
__global__ void __launch_bounds__(128) rix_count_kernel(const int32_t* __restrict__ idx, uint8_t* __restrict__ counts, uint4* __restrict__ visits,
                                                        int tiles, int32_t* __restrict__ zero, int nzero, int S, int NB, int Kb) {
    wait_for_previous_kernel();
    extern __shared__ __align__(16) uint32_t words[];
    const int qblk = blockIdx.x;
    const int64_t bp = blockIdx.y;
    const int32_t* tile = stage_rows(words, idx + (bp * S + static_cast<int64_t>(qblk) * kBlock) * Kb, NB, Kb);
    build_bitmap(words, tile, NB, Kb, qblk);
    if (visits && qblk < tiles) {
        uint4* vrow = visits + (bp * tiles + qblk) * tiles;
        for (int j = threadIdx.x; j <= qblk; j += blockDim.x) vrow[j] = reinterpret_cast<const uint4*>(words)[j];
    }
    if (!counts) {
        if (qblk == 0 && bp == 0)
            for (int i = threadIdx.x; i < nzero; i += blockDim.x) zero[i] = 0;
        return;
    }
    uint8_t* crow = counts + (bp * NB + qblk) * NB;
    for (int j = threadIdx.x; j <= qblk; j += blockDim.x) {
        const int c = __popc(words[j * 4]) + __popc(words[j * 4 + 1]) + __popc(words[j * 4 + 2]) + __popc(words[j * 4 + 3]);
        crow[j] = static_cast<uint8_t>(c);   // <= 128
    }
}

__global__ void rix_colscan_kernel(const uint8_t* __restrict__ counts, int32_t* __restrict__ blk_off,
                                   int32_t* __restrict__ totals, int64_t rows_bh, int NB) {
    wait_for_previous_kernel();
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= rows_bh * NB) return;
    const int64_t bp = t / NB;
    const int j = static_cast<int>(t % NB);
    int run = 0;
    for (int i = j; i < NB; ++i) {
        const int64_t at = (bp * NB + i) * NB + j;
        blk_off[at] = run;
        run += counts[at];
    }
    totals[t] = run;
}

__global__ void __launch_bounds__(1024) rix_rowscan_kernel(const int32_t* __restrict__ totals,
                                                           int32_t* __restrict__ row_ptr, int64_t n, int32_t* __restrict__ zero, int nzero) {
    wait_for_previous_kernel();
    if (zero)   // words a later kernel of the sequence wants to find zeroed
        for (int i = threadIdx.x; i < nzero; i += 1024) zero[i] = 0;
    __shared__ int64_t part[1024];
    const int tid = threadIdx.x;
    const int64_t per = (n + 1023) / 1024;
    const int64_t lo = tid * per, hi = (lo + per < n) ? lo + per : n;
    int64_t sum = 0;
    for (int64_t i = lo; i < hi; ++i) sum += totals[i];
    part[tid] = sum;
    __syncthreads();
    // Hillis-Steele inclusive scan over 1024 partials
    for (int off = 1; off < 1024; off <<= 1) {
        const int64_t v = (tid >= off) ? part[tid - off] : 0;
        __syncthreads();
        part[tid] += v;
        __syncthreads();
    }
    int64_t run = part[tid] - sum;
    for (int64_t i = lo; i < hi; ++i) {
        row_ptr[i] = static_cast<int32_t>(run);
        run += totals[i];
    }
    if (tid == 1023) row_ptr[n] = static_cast<int32_t>(part[1023]);
}

// Both scans in one launch where a single CTA has a thread for every column and the columns are short (B=3 S=1664 Hp=4, 156 columns of
// 13: the index 15.6 -> 10.7 us, with the count left to the selection).
constexpr int kRixOneScanCounts = 16384;   // (1024 columns of 64: 39 us for the index instead of 32)
inline bool one_scan(int64_t cols, int NB) { return cols <= 1024 && cols * NB <= kRixOneScanCounts; }
__global__ void __launch_bounds__(1024) rix_scan_kernel(const uint8_t* __restrict__ counts, int32_t* __restrict__ blk_off,
                                                        int32_t* __restrict__ row_ptr, int cols, int NB, int32_t* __restrict__ zero, int nzero) {
    wait_for_previous_kernel();
    if (zero)
        for (int i = threadIdx.x; i < nzero; i += 1024) zero[i] = 0;
    __shared__ int32_t part[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int run = 0;
    if (t < cols) {
        const int bp = t / NB, j = t % NB;
#pragma unroll 8
        for (int i = j; i < NB; ++i) {
            const int at = (bp * NB + i) * NB + j;
            blk_off[at] = run;
            run += counts[at];
        }
    }
    // exclusive scan of the totals over the CTA (fewer than 2^31 edges: checked at the entry)
    int incl = run;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += v;
    }
    if (lane == 31) part[warp] = incl;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; ++w) before += part[w];
    if (t < cols) row_ptr[t] = before + incl - run;
    if (t == cols - 1) row_ptr[cols] = before + incl;
}

__global__ void __launch_bounds__(128) rix_fill_kernel(const int32_t* __restrict__ idx, const int32_t* __restrict__ blk_off,
                                                       const int32_t* __restrict__ row_ptr, int32_t* __restrict__ col_q,
                                                       int32_t* __restrict__ edge_pos, int32_t* __restrict__ row_start, int tiles,
                                                       int S, int NB, int Kb) {
    wait_for_previous_kernel();
    extern __shared__ __align__(16) uint32_t words[];
    const int qblk = blockIdx.x;
    const int64_t bp = blockIdx.y;
    const int64_t row0 = bp * S + static_cast<int64_t>(qblk) * kBlock;
    int32_t* tile = stage_rows(words, idx + row0 * Kb, NB, Kb);
    build_bitmap(words, tile, NB, Kb, qblk);
    const int r = threadIdx.x;
    const int q = qblk * kBlock + r;
    int32_t* row = tile + r * Kb;   // the selections of row r; each is replaced by its edge position
    const int32_t* rp = row_ptr + bp * NB;
    const int32_t* bo = blk_off + (bp * NB + qblk) * NB;
    if (row_start && qblk == tiles)
        for (int j = r; j < NB; j += kBlock) row_start[bp * NB + j] = rp[j] + (j < tiles ? bo[j] : 0);
    const int w = r >> 5;
    const uint32_t below = (1u << (r & 31)) - 1u;
    for (int s = 0; s < Kb; ++s) {
        const int at = rotated_slot(s, r, Kb);
        const int j = row[at];
        int pos = -1;
        if (static_cast<unsigned>(j) < static_cast<unsigned>(NB) && j <= qblk) {
            int rank = __popc(words[j * 4 + w] & below);
            for (int ww = 0; ww < w; ++ww) rank += __popc(words[j * 4 + ww]);
            pos = rp[j] + bo[j] + rank;
            // (inside the row wherever the counts are those of these selections; no other index may lead out of col_q)
            if (pos < rp[j + 1]) col_q[pos] = q;
            else pos = -1;
        }
        row[at] = pos;
    }
    __syncthreads();
    // edge positions of the query block leave as one contiguous run
    const int4* src = reinterpret_cast<const int4*>(tile);
    int4* dst = reinterpret_cast<int4*>(edge_pos + row0 * Kb);
    for (int t = threadIdx.x; t < kBlock * Kb / 4; t += blockDim.x) dst[t] = src[t];
}

// Where query tiles first_tile .. begin in every row, for an index that was built without (one thread per row).
__global__ void __launch_bounds__(128) rix_row_start_kernel(const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ col_q,
                                                            int32_t* __restrict__ row_start, int64_t rows, int q0) {
    const int64_t r = static_cast<int64_t>(blockIdx.x) * 128 + threadIdx.x;
    if (r >= rows) return;
    int lo = row_ptr[r], hi = row_ptr[r + 1];   // query positions ascend inside a row
    while (lo < hi) {
        const int mid = lo + (hi - lo) / 2;
        if (col_q[mid] < q0) lo = mid + 1;
        else hi = mid;
    }
    row_start[r] = lo;
}

constexpr size_t kRixSmemCap = 160 * 1024;   // NB <= 2048 and Kb <= 128 need 96 KB; the attribute is set once, to the cap

}  // namespace

RixWorkspace carve_reverse_index(void* base, int64_t rows_bh, int NB) {
    RixWorkspace w;
    const size_t n2 = static_cast<size_t>(rows_bh) * NB * NB;
    size_t off = 0;
    w.counts = reinterpret_cast<uint8_t*>(static_cast<char*>(base) + off);
    off += static_cast<size_t>(round_up(static_cast<int64_t>(n2), 256));
    w.blk_off = reinterpret_cast<int32_t*>(static_cast<char*>(base) + off);
    off += static_cast<size_t>(round_up(static_cast<int64_t>(n2 * 4), 256));
    w.totals = reinterpret_cast<int32_t*>(static_cast<char*>(base) + off);
    off += static_cast<size_t>(round_up(static_cast<int64_t>(rows_bh) * NB * 4, 256));
    w.bytes = off;
    return w;
}

// Launch sequence shared with any other entry point that supplies its own scratch memory.
int reverse_index_launch(const int32_t* block_indices, int32_t* row_ptr, int32_t* col_q, int32_t* edge_pos,
                         int64_t rows_bh, int32_t S, int32_t Kb, void* scratch, cudaStream_t st, const RixExtras& x) {
    const int NB = S / kBlock;
    const RixWorkspace w = carve_reverse_index(scratch, rows_bh, NB);
    const dim3 grid(static_cast<unsigned>(NB), static_cast<unsigned>(rows_bh));
    const size_t smem = static_cast<size_t>(NB) * 16 + static_cast<size_t>(kBlock) * Kb * sizeof(int32_t);
    if (smem > kRixSmemCap || (reinterpret_cast<uintptr_t>(block_indices) & 15u) != 0 || (reinterpret_cast<uintptr_t>(edge_pos) & 15u) != 0)
        return FMSA_ERR_UNSUPPORTED;
    if (!ensure_smem_attr(reinterpret_cast<const void*>(rix_count_kernel), kRixSmemCap) ||
        !ensure_smem_attr(reinterpret_cast<const void*>(rix_fill_kernel), kRixSmemCap))
        return FMSA_ERR_CUDA;
    if (!x.counted)
        launch_chained(rix_count_kernel, grid, 128, smem, st, block_indices, w.counts, static_cast<uint4*>(x.visits), x.tiles, static_cast<int32_t*>(nullptr), 0, S, NB, Kb);
    const int64_t cols = rows_bh * NB;
    if (one_scan(cols, NB))
        launch_chained(rix_scan_kernel, 1, 1024, 0, st, w.counts, w.blk_off, row_ptr, static_cast<int>(cols), NB, x.zero, x.nzero);
    else
        launch_chained(rix_colscan_kernel, static_cast<unsigned>((cols + 127) / 128), 128, 0, st, w.counts, w.blk_off, w.totals, rows_bh, NB);
    if (!one_scan(cols, NB))
        launch_chained(rix_rowscan_kernel, 1, 1024, 0, st, w.totals, row_ptr, cols, x.zero, x.nzero);
    launch_chained(rix_fill_kernel, grid, 128, smem, st, block_indices, w.blk_off, row_ptr, col_q, edge_pos, x.row_start, x.tiles, S, NB, Kb);
    return check_launch();
}

int reverse_index_launches(int64_t rows_bh, int32_t S, const RixExtras& x) {
    const int NB = S / kBlock;
    return (x.counted ? 0 : 1) + (one_scan(rows_bh * NB, NB) ? 1 : 2) + 1;
}

int launch_tile_visits(const int32_t* block_indices, int64_t rows_bh, int32_t S, int32_t Kb, const RixExtras& x, cudaStream_t st) {
    const int NB = S / kBlock;
    const size_t smem = static_cast<size_t>(NB) * 16 + static_cast<size_t>(kBlock) * Kb * sizeof(int32_t);
    if (smem > kRixSmemCap || (reinterpret_cast<uintptr_t>(block_indices) & 15u) != 0) return FMSA_ERR_UNSUPPORTED;
    if (!ensure_smem_attr(reinterpret_cast<const void*>(rix_count_kernel), kRixSmemCap)) return FMSA_ERR_CUDA;
    launch_chained(rix_count_kernel, dim3(static_cast<unsigned>(x.tiles), static_cast<unsigned>(rows_bh)), 128, smem, st,
        block_indices, static_cast<uint8_t*>(nullptr), static_cast<uint4*>(x.visits), x.tiles, x.zero, x.nzero, S, NB, Kb);
    return check_launch();
}

size_t reverse_index_scratch_bytes(int64_t rows_bh, int32_t S) {
    return carve_reverse_index(nullptr, rows_bh, S / kBlock).bytes;
}

// -------------------------------------------------------------------------------------------
// Allocation-free variant: the scratch lives in the library image.
// -------------------------------------------------------------------------------------------
// Every GPU that loads the library holds these bytes until the process exits.
static __device__ __align__(256) unsigned char g_rix_static_scratch[FMSA_STATIC_SCRATCH_BYTES];

// In host code the array's name is only a handle for the runtime, not a device address, so the
// address is asked for once per device (with that device current) and cached.
static int static_scratch_address(void** out) {
    constexpr int kMaxDevices = 64;
    static void* cached[kMaxDevices] = {nullptr};
    static std::mutex guard;
    std::lock_guard<std::mutex> lock(guard);
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return FMSA_ERR_CUDA;
    if (cached[dev] == nullptr) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_rix_static_scratch) != cudaSuccess || p == nullptr) return FMSA_ERR_CUDA;
        cached[dev] = p;
    }
    *out = cached[dev];
    return FMSA_OK;
}

}  // namespace fmsa

extern "C" int fmsa_reverse_index_static(const int32_t* block_indices, int32_t* row_ptr, int32_t* col_q,
                                         int32_t* edge_pos, int64_t rows_bh, int32_t S, int32_t top_k_blocks,
                                         void* stream) {
    using namespace fmsa;
    FMSA_REQUIRE(block_indices && row_ptr && col_q && edge_pos);
    FMSA_REQUIRE(rows_bh > 0 && rows_bh <= 65535 && S > 0 && S % kBlock == 0);
    const int NB = S / kBlock;
    FMSA_REQUIRE(top_k_blocks >= 1 && top_k_blocks <= NB);
    FMSA_REQUIRE(rows_bh * static_cast<int64_t>(S) * top_k_blocks < 0x7fffffffLL);
    if (NB > 2048) return FMSA_ERR_UNSUPPORTED;
    // the problem must fit the built-in scratch; larger ones need fmsa_reverse_index and a workspace
    if (reverse_index_scratch_bytes(rows_bh, S) > static_cast<size_t>(FMSA_STATIC_SCRATCH_BYTES)) return FMSA_ERR_WORKSPACE;
    void* scratch = nullptr;
    const int rc = static_scratch_address(&scratch);
    if (rc != FMSA_OK) return rc;
    // Nothing in the scratch has to start at zero: every count, offset and total a kernel reads
    // was written earlier in the same call, so stale contents of a previous call are never seen.
    return reverse_index_launch(block_indices, row_ptr, col_q, edge_pos, rows_bh, S, top_k_blocks, scratch,
                                static_cast<cudaStream_t>(stream));
}

extern "C" int32_t fmsa_reverse_index_launches(int64_t rows_bh, int32_t S) {
    return rows_bh > 0 && S > 0 ? fmsa::reverse_index_launches(rows_bh, S, fmsa::RixExtras()) : 0;
}

extern "C" int fmsa_row_start(const int32_t* row_ptr, const int32_t* col_q, int64_t rows_bh, int32_t S, int32_t first_tile,
                              int32_t* row_start, void* stream) {
    using namespace fmsa;
    FMSA_REQUIRE(row_ptr && col_q && row_start && rows_bh > 0 && rows_bh <= 65535 && S > 0 && S % kBlock == 0 && first_tile >= 0);
    const int64_t rows = rows_bh * (S / kBlock);
    FMSA_REQUIRE(first_tile <= S / kBlock);
    rix_row_start_kernel<<<static_cast<unsigned>((rows + 127) / 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(row_ptr, col_q, row_start,
                                                                                                            rows, first_tile * kBlock);
    return check_launch();
}

extern "C" size_t fmsa_reverse_index_workspace_bytes(int64_t rows_bh, int32_t S) {
    if (rows_bh <= 0 || S <= 0 || S % fmsa::kBlock != 0) return 0;
    return fmsa::reverse_index_scratch_bytes(rows_bh, S);
}

extern "C" int fmsa_reverse_index(const int32_t* block_indices, int32_t* row_ptr, int32_t* col_q, int32_t* edge_pos,
                                  int64_t rows_bh, int32_t S, int32_t top_k_blocks, void* workspace,
                                  size_t workspace_bytes, void* stream) {
    using namespace fmsa;
    FMSA_REQUIRE(block_indices && row_ptr && col_q && edge_pos && workspace);
    FMSA_REQUIRE(rows_bh > 0 && rows_bh <= 65535 && S > 0 && S % kBlock == 0);
    const int NB = S / kBlock;
    FMSA_REQUIRE(top_k_blocks >= 1 && top_k_blocks <= NB);
    FMSA_REQUIRE(rows_bh * static_cast<int64_t>(S) * top_k_blocks < 0x7fffffffLL);
    if (NB > 2048) return FMSA_ERR_UNSUPPORTED;   // bitmap must fit in shared memory (NB*16 bytes)
    FMSA_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0);
    if (workspace_bytes < reverse_index_scratch_bytes(rows_bh, S)) return FMSA_ERR_WORKSPACE;
    return reverse_index_launch(block_indices, row_ptr, col_q, edge_pos, rows_bh, S, top_k_blocks, workspace,
                                static_cast<cudaStream_t>(stream));
}

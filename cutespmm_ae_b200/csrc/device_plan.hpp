// Kernel argument blocks and launcher prototypes shared by the C ABI and the kernel files.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

namespace cutespmm {

// Opts a kernel in to more than 48 KB of dynamic shared memory.  The attribute belongs to the (function, device)
// pair, so it is set once per device ordinal: a process that drives several GPUs configures each of them.
// (The kernel is a template argument, not a function argument: the table below must be one per kernel, and two
// instantiations of a kernel template share a function-pointer type.)
template <auto Kernel> cudaError_t allow_dynamic_smem(int bytes)
{
    constexpr int kMaxDevices = 64;
    static std::atomic<bool> done[kMaxDevices] = {};  // several threads may come here at once: each sets the same
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < kMaxDevices && done[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && dev >= 0 && dev < kMaxDevices) done[dev] = true;
    return e;
}

// Blocks of `threads` threads of a kernel that an SM holds: the same for every device of one model, so asked once per kernel.
// Several threads may come here at once: each asks for and stores the same.
template <auto Kernel> cudaError_t blocks_per_sm(int &n, int threads)
{
    static std::atomic<int> known{0};
    if ((n = known) != 0) return cudaSuccess;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, Kernel, threads, 0);
    if (e != cudaSuccess) return e;
    if (n < 1) n = 1;
    known = n;
    return cudaSuccess;
}

// Launches a kernel whose blocks may be set up while the kernel in front of it on the stream still runs (the kernel calls
// ptx::grid_wait before it depends on anything): back-to-back calls of a 5-us product are a launch latency shorter each.
template <class... Params, class... Args>
cudaError_t launch_overlapped(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args &&...args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// Arguments of the row-gather kernel.
struct RowsArgs {
    const uint32_t *row_ptr;   // M+1 offsets into pairs
    const void *pairs;         // nnz x {col, fp32 bits}
    const void *tiles;         // num_tiles x {row_begin, row_end, pair_begin, pair_end}
    const void *chunks;        // num_chunks x {row, j0, j1, slot}
    const void *long_rows;     // the whole list of long rows {row of C, slot0, slot1, -}, indexed by chunk_owner
    const uint32_t *chunk_owner;  // per scratch slot: index of the long row the chunk belongs to
    uint32_t *arrivals;        // per long row of the list, kArrivalStride apart, kRowSlabs counters: chunks finished so far (zero between launches)
    uint32_t *counters;        // balance of the blocks that left, then tiles dealt per column slab (kRowSlabs of them); zero between
                               // launches.  nullptr: tiles in fixed turns
    uint32_t num_tiles, num_chunks;
    uint32_t avg_row_nnz;      // nonzeros per row of the whole matrix (picks the kernel's tuning)
    uint32_t uneven;           // 1: the list has chunks, and the other rows are of very different lengths, too (is_uneven)
    uint32_t short_chunks;     // 1: a small job, its long rows are cut into pieces of tens of nonzeros
    const float *B;            // K x N window, leading dimension ldb
    float *C;                  // M x N window, leading dimension ldc
    float *scratch;            // partial sums, leading dimension ld_scratch
    uint64_t ldb, ldc, ld_scratch;
    uint32_t N;
    uint32_t num_rows;         // of the whole matrix
    uint32_t run_rows;         // rows come in aligned runs of this many (2 or 3) with the same columns; 0: they do not
    uint32_t dense_panels;     // 1: some panels of 16 rows are dense enough for the tensor cores: neighbouring rows share columns
    uint32_t early;            // 1: the plan's arrays never change, its first tiles can be fetched before the kernel in front is done
    uint32_t b_padded;         // 1: a row of B can be read up to N rounded up to four columns
    uint32_t slab_cols;        // set by launch_rows: columns per slab of blocks (a multiple of 4)
    uint32_t c_scalar;         // set by launch_rows: C is written column by column
    uint32_t *status;          // device status word: set to 1 when a bounded wait gives up
    const uint32_t *row_map;   // reordered plan: row r of the work lists is row row_map[r] of C (nullptr: identity)
};

cudaError_t launch_block_rows(const RowsArgs &a, bool aligned, int sm_count, cudaStream_t s);
cudaError_t launch_rows(const RowsArgs &a, int sm_count, cudaStream_t s);
// dst: rows x (N rounded up to 4) floats, 16-byte aligned
cudaError_t launch_pad_rows(const float *src, uint64_t ld_src, float *dst, uint64_t rows, uint32_t N, int sm_count, cudaStream_t s);

// Arguments of the SDDMM kernel (sddmm_kernel.cu): out[j] = (scale ? value of nonzero j : 1) * <X[row of j], Y[column of j]>.
struct SddmmArgs {
    const uint32_t *row_ptr;
    const void *pairs, *tiles, *chunks;  // the plan's nonzeros and its row-kernel work list over every row
    uint32_t num_tiles, num_chunks;
    const float *X, *Y;                  // M x N and K x N, row-major
    uint64_t ldx, ldy;
    float *out;                          // one value per nonzero, in the plan's storage order
    uint32_t N;
    uint32_t scale;                      // 1: multiply by the stored value of A
    uint32_t short_rows;                 // 1: fewer than four nonzeros per row that has any (picks the kernel's form)
    uint32_t early;                      // 1: the plan's arrays never change (RowsArgs::early)
    uint32_t vec4;                       // 1: X, Y and their leading dimensions (below 2^30) allow 16-byte loads
    uint32_t *status;                    // device status word: set to 1 when a bounded wait gives up
};
cudaError_t launch_sddmm(const SddmmArgs &a, int sm_count, cudaStream_t s);

// Arguments of the tensor-core brick kernel.
constexpr int kBrickWarps = 15;  // warps per block; each is an independent pipeline over its own brick range
struct BrickArgs {
    const uint32_t *cols;         // 8 columns per brick slot (+ readable slack of a few groups behind the end)
    const uint32_t *recs;         // brick records (map, flags, panel, values in fragment order): slot k at word k * kBrickRecWords
    const uint32_t *panel_first;  // per brick panel: slot of its first brick (a multiple of 4)
    const uint32_t *panel_last;   // per brick panel: one past the slot of its last brick
    uint32_t num_bricks, num_panels;
    uint32_t M, K;
    const float *B;
    float *C;
    uint64_t ldb, ldc;
    uint32_t N;
    uint32_t round_b;             // 1: round B to tf32 to nearest, 0: truncate
    uint32_t *status;             // device status word: set to 2 when a bounded wait gives up
    const uint32_t *row_map;      // reordered plan: row r of a panel is row row_map[r] of C (nullptr: identity)
};

cudaError_t launch_brick(const BrickArgs &a, int sm_count, cudaStream_t s);
int brick_launches(uint32_t N);  // kernels launch_brick queues for N columns
bool brick_supports(uint32_t N, uint64_t ldb, uint64_t ldc, const void *B, const void *C);

// Arguments of the tcgen05 slab kernel (128-row panels).
struct SlabArgs {
    const uint32_t *cols;         // 8 columns per step slot (+ readable slack)
    const uint32_t *recs;         // step records
    const uint32_t *rec_off;      // per step slot (+1) record offsets in 16-byte units (+ slack)
    const uint32_t *panel_first;  // per slab panel: slot of its first step (a multiple of 4)
    const uint32_t *panel_last;   // per slab panel: one past the slot of its last step
    const uint32_t *panel_ids;    // per slab panel: its 128-row panel index
    uint32_t num_panels;
    uint32_t M, K;
    const float *B;
    float *C;
    uint64_t ldb, ldc;
    uint32_t N;                   // a multiple of 128
    uint32_t *status;             // device status word: set to 3 when a bounded wait gives up
};
cudaError_t launch_slab(const SlabArgs &a, int sm_count, cudaStream_t s);
bool slab_supports(uint32_t N, uint64_t ldb, uint64_t ldc, const void *B, const void *C);

// ---- device side of plan creation (device_build.cu; device_plan.cu runs it) ----
struct Tile;
struct Chunk;
struct LongRow;
constexpr uint32_t kRowPtrSlack = 8;  // row pointers repeated behind the last one: a tile's copy starts and ends on 16-byte boundaries
// kDevPanelMax: nonzeros of a panel the shared-memory sort (and the largest hash set) takes.  kMaxCensusNnz: the same for
// the census of path auto, which looks at panels without long rows only: 16 rows of at most kMaxSplitNnz nonzeros.
constexpr uint32_t kDevPanelMax = 8192, kMaxCensusNnz = 6144;

constexpr uint32_t kTileSegmentRows = 512;   // rows a block of the list kernels looks at; a multiple of kPanelRows
constexpr uint32_t kSegmentEntries = 257;    // kMaxTileRows + 1: rows of a segment its first tile can start at

struct BuildTotals {  // one per plan creation, read by the host after the counting kernels
    uint32_t nnz, bad_rows, bad_cols, too_large;
    uint32_t tiles;
    uint32_t chunks, long_rows, brick_panels, brick_slots;  // in the order of the per-segment counters
    uint32_t brick_nnz_max, brick_cols_max;
    uint32_t filled_rows;  // rows that have nonzeros
    uint32_t unlike;  // bit 0: some odd row has other columns than the row in front of it, bit 1: some row not divisible by 3
    unsigned long long bricks, brick_cost, long_nnz, mid_nnz;
};
struct ListArgs {
    uint32_t M, num_segments;
    uint32_t split_nnz, tile_nnz, adaptive;
    uint32_t total_known;   // 1: `total` is the cost of the listed rows; 0: every row is listed, nnz + kRowCost * M
    uint64_t total;
    const unsigned long long *long_nnz;  // nonzeros in long rows, summed by the survey
    const uint8_t *path;   // per panel: 1 = not listed (nullptr: every row is)
    uint16_t *exits, *tile_counts;  // per segment and entry row: entry row of the next segment, tiles
    uint16_t *path_entry;   // per segment and entry row of its group: entry row of the segment ...
    uint32_t *path_tiles;   // ... and tiles of the group in front of it
    uint16_t *group_exit;   // per group and entry row: entry row of the next group, tiles
    uint32_t *group_tiles;
    uint2 *group_entry;     // per group: real entry row, its first tile
    uint32_t *seg_chunks, *seg_longs;  // per segment: counts, then offsets
    BuildTotals *totals;
    Tile *tiles;
    Chunk *chunks;
    LongRow *long_rows;
    uint32_t *owners;
};
struct CensusArgs {
    uint32_t M, num_panels;
    uint32_t force;         // 1: path brick, every panel that fits
    uint32_t split_nnz;
    float density;
    uint32_t most, table_words;
    uint32_t *ncols;        // per panel: distinct columns (of candidates)
    uint8_t *path;          // per panel: 1 = brick
    uint32_t *seg_panels, *seg_slots;
    BuildTotals *totals;
};
cudaError_t launch_lists_count(const uint32_t *row_ptr, const ListArgs &a, cudaStream_t s);
cudaError_t launch_lists_scan(const uint32_t *row_ptr, const ListArgs &a, uint32_t *counters, uint32_t how_many, cudaStream_t s);
cudaError_t launch_lists_write(const uint32_t *row_ptr, const ListArgs &a, cudaStream_t s);
cudaError_t launch_row_survey(const uint32_t *row_ptr, const uint32_t *cols, uint32_t M, BuildTotals *totals, int sm_count, cudaStream_t s);
cudaError_t launch_panel_census(const uint32_t *row_ptr, const uint32_t *cols, CensusArgs a, int sm_count, cudaStream_t s);
cudaError_t launch_brick_layout(uint32_t num_panels, const uint8_t *path, const uint32_t *ncols, const uint32_t *seg_panels, const uint32_t *seg_slots,
                                uint32_t num_segments, uint32_t *ids, uint32_t *first, uint32_t *last, cudaStream_t s);
cudaError_t launch_brick_fill(const uint32_t *row_ptr, const void *pairs, uint32_t M, const uint32_t *ids, const uint32_t *first_slot,
                              uint32_t num_brick_panels, const uint32_t *ncols, uint32_t nnz_max, uint32_t cols_max, uint32_t *bcols, uint32_t *brecs,
                              int sm_count, cudaStream_t s);
cudaError_t launch_pack(const uint32_t *row_ptr, const uint32_t *cols, const float *vals, uint32_t M, uint32_t K, uint32_t nnz, uint32_t *row_ptr_out,
                        void *pairs, uint32_t *bad, int sm_count, cudaStream_t s);
cudaError_t launch_set_values(void *pairs, const float *vals, const uint32_t *order, uint64_t nnz, int sm_count, cudaStream_t s);
cudaError_t launch_unpack(const void *pairs, uint32_t *cols, float *vals, uint64_t nnz, int sm_count, cudaStream_t s);
// the panel views (distinct columns per panel, ascending) and column ranges, when somebody asks for them
cudaError_t launch_panel_columns(const uint32_t *row_ptr, const void *pairs, uint32_t M, uint32_t num_panels, uint32_t *ncols,
                                 uint32_t *acols, int sm_count, cudaStream_t s);
cudaError_t launch_panel_max_col(const uint32_t *row_ptr, const void *pairs, uint32_t M, uint32_t num_panels, uint32_t *maxcol, int sm_count,
                                 cudaStream_t s);

}  // namespace cutespmm

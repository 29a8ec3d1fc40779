// Internal definition of a plan: the device-resident form of A plus the work lists of the two
// kernel families.  Host code only (no CUDA types) so the builder can be compiled and tested on a
// machine without a GPU.
#pragma once
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/cutespmm.h"

#ifdef __CUDACC__
#define CUTESPMM_HD __host__ __device__
#else
#define CUTESPMM_HD
#endif

namespace cutespmm {

constexpr uint32_t kPanelRows = 16;   // row-panel height; HRPB's TM (inc.h:18-20)
constexpr uint32_t kBlockCols = 16;   // active-column block width; HRPB's TK (inc.h:21-23)
constexpr uint32_t kBrickCols = 8;    // one tensor-core brick is 16 rows x 8 active columns (mma m16n8k8)
constexpr uint32_t kRowCost = 4;      // scheduling cost of a row besides its nonzeros (pointer loads, C store)
constexpr uint32_t kDefaultSplitNnz = 256;
constexpr uint32_t kDefaultTileCost = 512;
constexpr uint32_t kMaxTileRows = 256;   // rows of one scheduling tile (bounds the staged row-pointer slice)
constexpr uint32_t kMaxTilePairs = 640;  // nonzeros of one scheduling tile (bounds the staged pair slice)
// Adaptive sizing of the row kernel's work items (when the caller leaves split_nnz and tile_nnz at 0):
constexpr uint32_t kResidentTiles = 560;          // tiles aimed at for a small job: one wave of the kernel's deep tuning (148 SMs x 4 blocks) less 5 %
constexpr uint32_t kMinAdaptiveTileCost = 96;     // smallest tile it makes (8 warps x 12 cost units)
constexpr uint32_t kMaxAdaptiveTileCost = 1024;   // largest: beyond it the job is not small, tiles go back to the default cost
constexpr uint32_t kAdaptiveSplitDivisor = 8192;  // rows are cut from job cost / this nonzeros on: 256 from 2.1 M cost units
constexpr uint32_t kMinAdaptiveSplitNnz = 128;    // ... but never from fewer than this
constexpr uint64_t kMidJobCost = 8u << 20;        // jobs up to this with an eighth of their nonzeros in long rows: cut from 128 on
constexpr uint32_t kWideTileRowNnz = 12;          // nonzeros per row from which a large job's tiles are larger:
constexpr uint32_t kWideTileCost = 768, kMixedTileCost = 640;  // ... and with an eighth of the nonzeros in long rows
constexpr uint32_t kMinChunkNnz = 32;             // smallest piece of a cut row
constexpr uint32_t kMaxSplitNnz = 384;   // a row must fit a tile together with a part-filled one
constexpr uint32_t kScratchCols = 512;  // widest N one launch handles; wider products run in column windows
constexpr uint32_t kRowSlabs = kScratchCols / 256;  // column slabs of a launch of the row kernel, which span 256 columns wherever one is not enough
// Words from one long row's arrival counters, one per column slab, to the next one's: two rows share a 128-byte line, packed 16 rows
// would (R-MAT 2^17 N = 64 47.4 -> 47.6 us, 2^16 28.4 -> 28.5).
constexpr uint32_t kArrivalStride = 16;
static_assert(kRowSlabs <= kArrivalStride);

// One nonzero as the row kernel reads it: column index and fp32 bit pattern side by side (8 bytes,
// one coalesced 64-bit load per lane).
struct Pair {
    uint32_t col;
    uint32_t val_bits;
};

// A scheduling tile of the row kernel: rows [row_begin, row_end) whose nonzeros are pairs
// [pair_begin, pair_end); at most kMaxTileRows rows and kMaxTilePairs nonzeros, no long row inside.
struct Tile {
    uint32_t row_begin, row_end, pair_begin, pair_end;
};

// Sizes of the row kernel's work items for a list whose rows cost `total` (nonzeros + kRowCost per row): used as they
// are by the host builder and by the device builder's kernels.
//
// The default sizes (tiles of cost 512, chunks of 256 nonzeros) keep the per-item overhead small when the grid is
// many waves long.  A small job is a handful of memory latencies long, and then the longest chain of dependent
// gathers of one warp IS the run time: a 256-nonzero chunk is 64 steps of four loads, about 30 us, when the
// rest of a 200 000-nonzero matrix is done in 10.  So the work is cut finer the smaller the job: tiles so that
// one resident wave of blocks holds them all, rows cut from a shorter length on (not below 128: a piece costs
// about eight latencies of its own -- descriptor, pairs, arrival count, the sum -- so shorter rows are quicker
// whole), and a cut row into pieces of about sqrt(length / 2) nonzeros: the chain is a piece's gathers followed
// by the sum of the pieces, the sum runs a few slots per step, and that length makes the two about equal.
//
// Larger jobs: a graph with much of its nonzeros in long rows is cut finer up to kMidJobCost (R-MAT 2^17 N = 32 56 -> 41 us,
// 2^18 N = 64 118 -> 99: a chunk of 256 is still a visible part of the run; beyond, N = 128 loses what N = 32 gains), and
// rows of a dozen nonzeros and more get larger tiles (elasticity40 N = 32 41 -> 37 us: fewer starts per nonzero).
struct ItemSizes {
    uint32_t split;      // rows longer than this are cut into chunks
    uint32_t target;     // cost at which a tile is closed
    bool latency_bound;  // pieces of sqrt(length / 2)
};
// nnz, M: of the whole matrix; long_nnz: its nonzeros in rows longer than kDefaultSplitNnz
CUTESPMM_HD inline ItemSizes item_sizes(uint64_t total, uint64_t nnz, uint64_t M, uint64_t long_nnz, uint32_t split_nnz, uint32_t tile_nnz, bool adaptive)
{
    ItemSizes s{split_nnz, tile_nnz, false};
    if (!adaptive) return s;
    if (total / kResidentTiles <= kMaxAdaptiveTileCost) {
        const uint64_t t = total / kResidentTiles;
        s.target = (uint32_t)(t > kMinAdaptiveTileCost ? t : kMinAdaptiveTileCost);
    } else if (nnz >= kWideTileRowNnz * M) {
        s.target = long_nnz * 8 >= nnz ? kMixedTileCost : kWideTileCost;
    }
    if (total / kAdaptiveSplitDivisor < s.split) {
        s.latency_bound = true;
        const uint64_t t = total / kAdaptiveSplitDivisor;
        s.split = (uint32_t)(t > kMinAdaptiveSplitNnz ? t : kMinAdaptiveSplitNnz);
    } else if (total < kMidJobCost && long_nnz * 8 >= nnz && s.split > kMinAdaptiveSplitNnz) {
        s.split = kMinAdaptiveSplitNnz;
    }
    return s;
}
// Rows are of very different lengths: an eighth of the nonzeros (mid_nnz) sits in rows of more than twice the mean and more than 32,
// those beyond kDefaultSplitNnz left out, which are cut up anyway, or a quarter in the latter (long_nnz).  R-MAT graphs of up to 20
// edges per node and side hold 25 to 43 % in the former, denser ones 50 to 78 % in the latter.  A few long rows in a matrix of short
// ones do not make it uneven.
CUTESPMM_HD inline bool mid_row(uint32_t len, uint64_t nnz, uint64_t M) { return len > 32 && len <= kDefaultSplitNnz && len * M > 2 * nnz; }
CUTESPMM_HD inline bool is_uneven(uint64_t mid_nnz, uint64_t long_nnz, uint64_t nnz) { return mid_nnz > nnz / 8 || long_nnz > nnz / 4; }
// nonzeros per chunk of a row of `len` nonzeros that is being cut
CUTESPMM_HD inline uint32_t piece_length(const ItemSizes &s, uint32_t len)
{
    if (!s.latency_bound) return s.split;
    uint32_t r = 1;
    while ((uint64_t)r * r * 2 < len) ++r;  // ceil(sqrt(len / 2)): a latency-bound job has fewer than 2.1 M nonzeros, about 1 000 steps at most
    if (r < kMinChunkNnz) r = kMinChunkNnz;
    return r < s.split ? r : s.split;
}

constexpr uint32_t kMinBrickPanels = 4440;  // path auto: fewer dense panels than two per warp of a full brick grid go to the row kernel
constexpr uint32_t kPanelTooLarge = 0xffffffffu;  // column count of a panel the device builder did not analyse

// A chunk of a long row: nonzeros [j0, j1) of `row`; its partial result is row `slot` of the scratch.
struct Chunk {
    uint32_t row, j0, j1, slot;
};
// A long row: C[row] = sum of scratch rows [slot0, slot1), added in that order.
struct LongRow {
    uint32_t row, slot0, slot1, pad;
};

// The brick kernel reads one flat stream of bricks (16 rows x 8 active columns each), panel after
// panel.  Brick k owns columns brick_cols[8k .. 8k+8) and the record that starts at 16-byte unit
// brick_rec_off[k] of brick_recs:
//     words 0-3   occupancy map, bit (r*8 + c) set when A[row r of the panel][column c of the brick] is stored
//     word  4     bit 0: last brick of its panel
//     word  5     panel index (rows 16*panel .. 16*panel+15)
//     words 6-7   0
//     words 8-135 the whole 16 x 8 brick (fp32, unrounded), zeros included, in the order the MMA wants it: word
//                 8 + 4*lane + i is A-fragment register i of that lane (brick_frag_index below), so a lane expands
//                 nothing: it loads its four values with one 128-bit read
// Every slot has a record of kBrickRecWords words (empty slots: zeros), brick k at word k * kBrickRecWords.
// (A packed record -- map plus the stored values only, expanded by popcounts as the reference does,
// kernel.cu:20-27 -- is a quarter of the size but was measured 5-11 % slower: the expansion is 50 dependent
// instructions per brick in a kernel that is bound by instruction latency, not by bytes.)
constexpr uint32_t kBrickRecHeaderWords = 8;
constexpr uint32_t kBrickRecWords = kBrickRecHeaderWords + 128;
// mma.m16n8k8 row-major A fragment: lane (g = lane / 4, t = lane % 4) holds a0 = A[g][t], a1 = A[g+8][t],
// a2 = A[g][t+4], a3 = A[g+8][t+4].  Position of element (row r, column c) of a brick in the dense record.
constexpr uint32_t brick_frag_index(uint32_t r, uint32_t c) { return ((r & 7u) * 4u + (c & 3u)) * 4u + (r >> 3) + 2u * (c >> 2); }
constexpr uint32_t kSlabRows = 128;      // rows of a slab panel (the M of one tcgen05.mma)
constexpr uint32_t kSlabMaxVals = 192;   // values one step record may hold (bounds the shared-memory stage)
constexpr uint32_t kSlabMaxRows = 32;    // rows one step record may list (one builder lane each)
constexpr uint32_t kSlabRecHeaderWords = 8;
constexpr uint32_t kSlabRecMaxWords = kSlabRecHeaderWords + kSlabMaxRows + kSlabMaxVals;

struct HostPlan {
    uint64_t M = 0, K = 0, nnz = 0;
    cutespmm_options_t opts{};
    bool device_built = false;  // the nonzeros were packed on the device; the host holds row pointers and work lists only
    bool values_on_device = false;  // cutespmm_plan_set_values replaced the values on the device: the host copy in `pairs` is stale
    bool adaptive_tiling = false;  // the caller left split_nnz and tile_nnz at 0: small jobs get smaller tiles and chunks

    // ---- row reordering (CUTESPMM_REORDER_CLUSTER_ROWS): row r of everything below is row row_map[r] of the caller's
    // matrix, and the kernels write its result to that row of C; empty = identity ----
    std::vector<uint32_t> row_map;

    // ---- row kernel ----
    std::vector<uint32_t> row_ptr;       // M+1, offsets into pairs
    std::vector<Pair> pairs;             // nnz
    std::vector<Tile> tiles;
    std::vector<uint8_t> row_path;       // per panel: 0 = rows kernel, 1 = brick kernel
    std::vector<Chunk> chunks;
    std::vector<LongRow> long_rows;

    bool uneven = false;                 // rows of very different lengths (is_uneven)
    uint64_t filled_rows = 0;            // rows that have nonzeros
    uint32_t run_rows = 0;               // rows come in aligned runs of 3 or 2 with the same columns (0: they do not)

    // ---- panel analysis (HRPB-compatible view) ----
    std::vector<uint32_t> blocked_row_ptr;  // num_panels+1
    std::vector<uint32_t> active_cols;      // per panel ascending distinct columns, zero-padded to x16

    // largest column index of every 16-row panel (0 for an empty panel): which rows of B a block of rows needs, for
    // the host-buffer call that lets rows of C leave while later rows of B still arrive
    std::vector<uint32_t> panel_max_col;

    // ---- row kernel over every row (used when a product's N does not fit the brick kernel) ----
    std::vector<Tile> tiles_all;
    std::vector<Chunk> chunks_all;
    std::vector<LongRow> long_rows_all;

    // ---- brick kernel ----
    std::vector<uint32_t> brick_cols;     // 8 per brick (a short last brick repeats its last column)
    std::vector<uint32_t> brick_recs;     // records, see above
    std::vector<uint32_t> brick_rec_off;  // per brick slot (+1) the record offset in 16-byte units
    // Brick slots: every panel's bricks are followed by empty slots up to a multiple of 4, so a
    // panel starts on a group-of-4 boundary of brick_cols / brick_rec_off.
    std::vector<uint32_t> panel_first_brick;  // per brick panel: slot of its first brick (multiple of 4)
    std::vector<uint32_t> panel_last_brick;   // per brick panel: one past the slot of its last brick
    uint64_t num_bricks = 0;
    uint64_t brick_panels = 0;
    std::vector<uint32_t> brick_panel_ids;    // device-built plans: the panel index of every brick panel, ascending
    uint64_t brick_slots = 0;                 // slots of the brick stream (bricks plus the empty slots that pad panels to groups of 4)

    // ---- slab kernel (tcgen05): 128-row panels, one record per step of 8 active columns ----
    // Step t owns columns slab_cols[8t .. 8t+8) and the record at 16-byte unit slab_rec_off[t] of slab_recs:
    //     word 0      number of rows with a nonzero in this step | (last step of its panel) << 16
    //     word 1      128-row panel index
    //     word 2      number of values stored (<= kSlabMaxVals), word 3: 0
    //     words 4-7   128-bit map of the rows that have an entry
    //     words 8..   one entry per such row, in row order: row in panel | 8-bit column mask << 8 | index of its first value << 16
    //                 (padded to a multiple of 4 entries), then the values in (row, column) order, padded to x4
    // A step with more than kSlabMaxRows rows or kSlabMaxVals values is stored as several steps over the same 8 columns.
    // Every panel's steps are followed by empty slots up to a multiple of 4 (group-aligned metadata).
    std::vector<uint32_t> slab_cols, slab_recs, slab_rec_off;
    std::vector<uint32_t> slab_first, slab_last;  // per 128-row panel with nonzeros: slot range of its steps
    std::vector<uint32_t> slab_ids;               // ... and its panel index (rows 128*id .. 128*id+127)
    std::vector<uint8_t> slab_path;               // per 128-row panel: 1 = executed by the slab kernel
    uint64_t slab_steps = 0, slab_panels = 0;

    uint64_t num_panels() const { return (M + kPanelRows - 1) / kPanelRows; }
};

// Validates the CSR input and fills every host-side member of `p`.  Returns a cutespmm_status_t;
// on failure `err` holds the message.
int build_host_plan(HostPlan &p, uint64_t M, uint64_t K, const uint64_t *rowPtr, const uint32_t *cols,
                    const float *vals, const cutespmm_options_t *opts, std::string &err);

// The options of a plan that is built on the device, checked and with the defaults filled in (p.opts, p.adaptive_tiling).
int check_device_options(HostPlan &p, uint64_t M, uint64_t K, const cutespmm_options_t *opts, std::string &err);

// HostPlan::uneven and ::filled_rows of a matrix whose row pointers are on the host.
void survey_rows(HostPlan &p);

// HostPlan::run_rows of a matrix whose pairs are on the host.
uint32_t find_row_runs(const HostPlan &p);

// Rebuilds CSR from the packed arrays (rows-kernel part from pairs, brick part from maps + values).
void decode_host_plan(const HostPlan &p, uint64_t *rowPtr, uint32_t *cols, float *vals);

int partition_rows(uint64_t M, const uint64_t *rowPtr, uint32_t nparts, uint32_t align_rows, uint32_t row_cost,
                   uint64_t *bounds, std::string &err);

}  // namespace cutespmm

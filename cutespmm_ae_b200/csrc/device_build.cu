// Kernels of cutespmm_plan_create_device (device_plan.cu): CSR that already lives on the GPU becomes a plan without its
// nonzeros or row pointers visiting the host -- the row kernel's work lists, the panel census that picks each panel's
// kernel, the tensor-core bricks and the packed (column, value) pairs.  The reference preprocesses on the host only
// (HRPB, data.cu:80-335) and its caller uploads the result.  Every kernel here reads each array it needs about once and
// is short (5-40 us at 2 M nonzeros); what a plan costs is their number and the two host round trips between them.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "device_plan.hpp"
#include "plan.hpp"
#include "ptx.cuh"

namespace cutespmm {

namespace {

constexpr unsigned kFullMask = 0xffffffffu;

// ---- panel analysis: the distinct columns of every 16-row panel, ascending --------------------------------------
// The device counterpart of HRPB's per-panel column census (reference data.cu:116-209, a K-sized flag array per
// thread): one block per panel sorts the panel's column indices in shared memory (bitonic) and compacts the distinct
// ones into acols[row_ptr[first row of the panel] ...] -- a panel has at most as many distinct columns as nonzeros,
// so the panel's own nonzero range is room enough.  Panels with more than kDevPanelMax nonzeros are left out
// (ncols = kPanelTooLarge): they hold a long row and stay with the row kernel.
__global__ void __launch_bounds__(256) panel_columns_kernel(const uint32_t *__restrict__ row_ptr, const uint2 *__restrict__ pairs, uint32_t M,
                                                            uint32_t num_panels, uint32_t *__restrict__ ncols,
                                                            uint32_t *__restrict__ acols)
{
    extern __shared__ uint32_t buf[];  // kDevPanelMax column indices
    __shared__ uint32_t warp_sums[8];
    __shared__ uint32_t running;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (uint32_t q = blockIdx.x; q < num_panels; q += gridDim.x) {
        const uint32_t r0 = q * kPanelRows, r1 = min(M, r0 + kPanelRows);
        const uint32_t j0 = __ldg(row_ptr + r0), n = __ldg(row_ptr + r1) - j0;
        if (n == 0 || n > kDevPanelMax) {
            if (tid == 0) ncols[q] = n == 0 ? 0u : kPanelTooLarge;
            continue;
        }
        uint32_t size = 32;
        while (size < n) size <<= 1;
        for (uint32_t i = tid; i < size; i += blockDim.x) buf[i] = i < n ? __ldg(&pairs[j0 + i].x) : 0xffffffffu;
        if (tid == 0) running = 0;
        __syncthreads();
        for (uint32_t k = 2; k <= size; k <<= 1)
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                for (uint32_t i = tid; i < size; i += blockDim.x) {
                    const uint32_t x = i ^ j;
                    if (x > i) {
                        const uint32_t a = buf[i], b = buf[x];
                        if ((a > b) == ((i & k) == 0)) {
                            buf[i] = b;
                            buf[x] = a;
                        }
                    }
                }
                __syncthreads();
            }
        // compact the distinct values, in order: rank = number of distinct values in front
        for (uint32_t base = 0; base < n; base += blockDim.x) {
            const uint32_t i = base + tid;
            const bool first = i < n && (i == 0 || buf[i] != buf[i - 1]);
            const unsigned ballot = __ballot_sync(kFullMask, first);
            if (lane == 0) warp_sums[warp] = __popc(ballot);
            __syncthreads();
            uint32_t off = running;
            for (uint32_t w = 0; w < warp; ++w) off += warp_sums[w];
            if (first) acols[j0 + off + __popc(ballot & ((1u << lane) - 1u))] = buf[i];
            __syncthreads();
            if (tid == 0) {
                uint32_t t = 0;
                for (uint32_t w = 0; w < blockDim.x / 32; ++w) t += warp_sums[w];
                running += t;
            }
            __syncthreads();
        }
        if (tid == 0) ncols[q] = running;
        __syncthreads();
    }
}

// maxcol[q] = largest column index among the nonzeros of 16-row panel q (0 when it has none); one warp per panel
__global__ void __launch_bounds__(256) panel_max_col_kernel(const uint32_t *__restrict__ row_ptr, const uint2 *__restrict__ pairs, uint32_t M,
                                                            uint32_t num_panels, uint32_t *__restrict__ maxcol)
{
    const uint32_t lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x / 32);
    for (uint32_t q = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); q < num_panels; q += warps) {
        const uint32_t r0 = q * kPanelRows, r1 = min(M, r0 + kPanelRows);
        const uint32_t j0 = __ldg(row_ptr + r0), j1 = __ldg(row_ptr + r1);
        uint32_t m = 0;
        for (uint32_t j = j0 + lane; j < j1; j += 32) m = max(m, __ldg(&pairs[j].x));
        for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(kFullMask, m, o));
        if (lane == 0) maxcol[q] = m;
    }
}

// ---- work lists of the row kernel ----------------------------------------------------------------------------------
// The tiles, chunks and long rows that build_tiles (plan.cpp) cuts, cut in parallel.  Where a tile ends depends on where
// it starts, so the tiles of a segment of rows depend on the row its first tile starts at -- but a tile has at most
// kMaxTileRows rows, so there are only kMaxTileRows + 1 such rows.  The counting kernel follows the chain of tiles from
// each of them at once (a thread per entry row), which gives the row the next segment is entered at and the number of
// tiles; the tables of 32 segments are composed into one, a single block walks those, and the writing kernel cuts every
// segment again from the one entry row that is real.  512 rows per segment: 2048 gave R-MAT 2^17 64 blocks and 76 us for
// counting and writing.  (The row pointers used to visit the host, which cut the lists there: for
// R-MAT 2^17, 1.9 M nonzeros, copies and host loops of 2-6 ms against 20 us.)
constexpr int kListThreads = 288;  // >= kEntries
constexpr uint32_t kEntries = kSegmentEntries;
static_assert(kEntries == kMaxTileRows + 1 && kTileSegmentRows % kPanelRows == 0, "entry rows");
static_assert(kListThreads >= (int)kEntries && kListThreads % 32 == 0, "a thread per entry row");
constexpr uint32_t kSegmentView = kTileSegmentRows + kMaxTileRows;  // rows a segment's last tile may reach

struct SegmentView {
    uint32_t rp[kSegmentView + 1];           // row pointers of rows [first, first + n]
    uint32_t special[kSegmentView / 32 + 1];  // bit r: row is long, or not in this list
    uint16_t next[kTileSegmentRows];         // where the tile that starts at a row ends (special row: the next row that is not)
    uint32_t n;
};

__device__ __forceinline__ bool is_special(const SegmentView &v, uint32_t r) { return (v.special[r >> 5] >> (r & 31)) & 1u; }
// first row in [r, n) whose special bit is `want`; n when there is none
__device__ __forceinline__ uint32_t find_row(const SegmentView &v, uint32_t r, uint32_t limit, bool want)
{
    while (r < limit) {
        const uint32_t w = (want ? v.special[r >> 5] : ~v.special[r >> 5]) >> (r & 31);
        if (w) return min(limit, r + __ffs(w) - 1);
        r = (r | 31) + 1;
    }
    return limit;
}

// Whole block: the rows of segment `seg` in shared memory and the tile ends of each as a start.  Returns whether this
// thread met row pointers that decrease or pass nnz.
__device__ __forceinline__ bool load_segment(SegmentView &v, const uint32_t *__restrict__ row_ptr, const ListArgs &a, const ItemSizes &sizes, uint32_t seg,
                                             uint32_t nnz)
{
    const uint32_t first = seg * kTileSegmentRows, n = min(a.M - first, kSegmentView);
    for (uint32_t r = threadIdx.x; r <= n; r += kListThreads) v.rp[r] = __ldg(row_ptr + first + r);
    if (threadIdx.x == 0) v.n = n;
    __syncthreads();
    bool bad = false;
    for (uint32_t b = threadIdx.x & ~31u; b < n; b += kListThreads) {
        const uint32_t r = b + (threadIdx.x & 31);
        bool sp = false;
        if (r < n) {
            const uint32_t p0 = v.rp[r], p1 = v.rp[r + 1];
            bad |= p1 < p0 || p1 > nnz;
            sp = (a.path && __ldg(a.path + (first + r) / kPanelRows)) || (p1 >= p0 && p1 - p0 > sizes.split);
        }
        const unsigned m = __ballot_sync(kFullMask, sp);
        if ((threadIdx.x & 31) == 0) v.special[b >> 5] = m;
    }
    __syncthreads();
    for (uint32_t r = threadIdx.x; r < min(n, kTileSegmentRows); r += kListThreads) {
        uint32_t e;
        if (is_special(v, r)) {
            e = find_row(v, r + 1, n, false);
        } else {
            // smallest e whose tile [r, e) has cost >= target, or whose next row would not fit the tile any more
            uint32_t lo = r + 1, hi = find_row(v, r + 1, min(n, r + kMaxTileRows), true);
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (v.rp[mid] - v.rp[r] + kRowCost * (mid - r) >= sizes.target || v.rp[mid + 1] - v.rp[r] > kMaxTilePairs) hi = mid;
                else lo = mid + 1;
            }
            e = max(lo, r + 1);
        }
        v.next[r] = (uint16_t)e;
    }
    __syncthreads();
    return bad;
}

__device__ __forceinline__ ItemSizes list_sizes(const ListArgs &a, uint32_t nnz)
{
    return item_sizes(a.total_known ? a.total : (uint64_t)nnz + (uint64_t)kRowCost * a.M, nnz, a.M, *a.long_nnz, a.split_nnz, a.tile_nnz, a.adaptive != 0);
}
// pieces of row r when it is long and in the list
__device__ __forceinline__ uint32_t pieces_of(const SegmentView &v, const ListArgs &a, const ItemSizes &sizes, uint32_t first, uint32_t r)
{
    const uint32_t len = v.rp[r + 1] - v.rp[r];
    if (v.rp[r + 1] < v.rp[r] || len <= sizes.split || (a.path && __ldg(a.path + (first + r) / kPanelRows))) return 0;
    const uint32_t piece = piece_length(sizes, len);
    return (len + piece - 1) / piece;
}

__global__ void __launch_bounds__(kListThreads) lists_count_kernel(const uint32_t *__restrict__ row_ptr, ListArgs a)
{
    ptx::grid_release();  // the census, next on the stream, needs nothing of this kernel: it runs beside it
    ptx::grid_wait();
    __shared__ SegmentView v;
    __shared__ uint32_t chunks, longs, wrong;
    const uint32_t seg = blockIdx.x, first = seg * kTileSegmentRows, nnz = __ldg(row_ptr + a.M);
    const ItemSizes sizes = list_sizes(a, nnz);
    if (threadIdx.x == 0) chunks = longs = wrong = 0;
    bool bad = load_segment(v, row_ptr, a, sizes, seg, nnz);
    bad |= seg == 0 && v.rp[0] != 0;
    const uint32_t rows = min(v.n, kTileSegmentRows);
    for (uint32_t r = threadIdx.x; r < rows; r += kListThreads)
        if (is_special(v, r)) {
            const uint32_t k = pieces_of(v, a, sizes, first, r);
            if (k) {
                atomicAdd(&chunks, k);
                atomicAdd(&longs, 1u);
            }
        }
    if (bad) wrong = 1;
    if (threadIdx.x < kEntries) {
        uint32_t r = threadIdx.x, tiles = 0;
        while (r < rows) {
            tiles += !is_special(v, r);
            r = v.next[r];
        }
        a.exits[(size_t)seg * kEntries + threadIdx.x] = (uint16_t)(r > kTileSegmentRows ? r - kTileSegmentRows : 0u);
        a.tile_counts[(size_t)seg * kEntries + threadIdx.x] = (uint16_t)tiles;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        a.seg_chunks[seg] = chunks;
        a.seg_longs[seg] = longs;
        if (wrong) atomicOr(&a.totals->bad_rows, 1u);
    }
}

// One block per group of kGroup segments, a thread per entry row of the group's first: the entry row of every segment
// and the tiles in front of it, were the group entered there; and the group's own exit and tiles.
constexpr uint32_t kGroup = 32;
__global__ void __launch_bounds__(kListThreads) lists_compose_kernel(ListArgs a)
{
    ptx::grid_wait();
    ptx::grid_release();
    __shared__ uint16_t exits[kGroup * kEntries], counts[kGroup * kEntries];
    const uint32_t s0 = blockIdx.x * kGroup, n = min(kGroup, a.num_segments - s0);
    for (uint32_t i = threadIdx.x; i < n * kEntries; i += kListThreads) {
        exits[i] = a.exits[(size_t)s0 * kEntries + i];
        counts[i] = a.tile_counts[(size_t)s0 * kEntries + i];
    }
    __syncthreads();
    const uint32_t e = threadIdx.x;
    if (e >= kEntries) return;
    uint32_t at = e, tiles = 0;
    for (uint32_t k = 0; k < n; ++k) {
        a.path_entry[(size_t)(s0 + k) * kEntries + e] = (uint16_t)at;
        a.path_tiles[(size_t)(s0 + k) * kEntries + e] = tiles;
        tiles += counts[k * kEntries + at];
        at = exits[k * kEntries + at];
    }
    a.group_exit[(size_t)blockIdx.x * kEntries + e] = (uint16_t)at;
    a.group_tiles[(size_t)blockIdx.x * kEntries + e] = tiles;
}

// Block 0 walks the groups: the row each is really entered at and the number of its first tile.  Block 1 + i turns the
// i-th per-segment counter into exclusive sums, in place.  The sums go to the totals.
constexpr uint32_t kChainBatch = 16;  // groups whose tables are in shared memory at a time
__global__ void __launch_bounds__(1024) lists_scan_kernel(const uint32_t *__restrict__ row_ptr, ListArgs a, uint32_t *__restrict__ counters)
{
    ptx::grid_wait();
    ptx::grid_release();
    __shared__ uint32_t sums[32];
    __shared__ uint16_t exits[kChainBatch * kEntries];
    __shared__ uint32_t counts[kChainBatch * kEntries];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (blockIdx.x == 0) {
        uint32_t entry = 0, tiles = 0;
        const uint32_t groups = (a.num_segments + kGroup - 1) / kGroup;
        for (uint32_t g0 = 0; g0 < groups; g0 += kChainBatch) {
            const uint32_t n = min(kChainBatch, groups - g0);
            for (uint32_t i = tid; i < n * kEntries; i += 1024) {
                exits[i] = a.group_exit[(size_t)g0 * kEntries + i];
                counts[i] = a.group_tiles[(size_t)g0 * kEntries + i];
            }
            __syncthreads();
            if (tid == 0)
                for (uint32_t k = 0; k < n; ++k) {
                    a.group_entry[g0 + k] = make_uint2(entry, tiles);
                    tiles += counts[k * kEntries + entry];
                    entry = exits[k * kEntries + entry];
                }
            __syncthreads();
        }
        if (tid == 0) {
            a.totals->tiles = tiles;
            a.totals->nnz = __ldg(row_ptr + a.M);
        }
        return;
    }
    uint32_t *v = counters + (size_t)(blockIdx.x - 1) * a.num_segments;
    uint32_t running = 0;
    for (uint32_t b = 0; b < a.num_segments; b += 1024) {
        const uint32_t x = b + tid < a.num_segments ? v[b + tid] : 0u;
        uint32_t incl = x;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        if (lane == 31) sums[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            uint32_t t = sums[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFullMask, t, o);
                if (lane >= (uint32_t)o) t += y;
            }
            sums[lane] = t;
        }
        __syncthreads();
        if (b + tid < a.num_segments) v[b + tid] = running + (warp ? sums[warp - 1] : 0u) + incl - x;
        running += sums[31];
        __syncthreads();
    }
    if (tid == 0) (&a.totals->chunks)[blockIdx.x - 1] = running;
}

__global__ void __launch_bounds__(kListThreads) lists_write_kernel(const uint32_t *__restrict__ row_ptr, ListArgs a)
{
    ptx::grid_release();  // reads the counts the host has waited for and writes lists nobody else touches: runs beside pack_kernel
    __shared__ SegmentView v;
    __shared__ uint16_t starts[kTileSegmentRows];
    __shared__ uint32_t num_starts, warp_longs[kListThreads / 32], warp_chunks[kListThreads / 32];
    const uint32_t seg = blockIdx.x, first = seg * kTileSegmentRows, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nnz = __ldg(row_ptr + a.M);
    const ItemSizes sizes = list_sizes(a, nnz);
    load_segment(v, row_ptr, a, sizes, seg, nnz);
    const uint32_t rows = min(v.n, kTileSegmentRows);
    const uint2 group = a.group_entry[seg / kGroup];  // the group's real entry row, tiles in front of the group
    if (tid == 0) {
        uint32_t k = 0;
        for (uint32_t r = a.path_entry[(size_t)seg * kEntries + group.x]; r < rows; r = v.next[r])
            if (!is_special(v, r)) starts[k++] = (uint16_t)r;
        num_starts = k;
    }
    // long rows and their chunks, in row order
    uint32_t lr = __ldg(a.seg_longs + seg), ck = __ldg(a.seg_chunks + seg);
    for (uint32_t b = 0; b < rows; b += kListThreads) {
        const uint32_t r = b + tid;
        const uint32_t pieces = r < rows && is_special(v, r) ? pieces_of(v, a, sizes, first, r) : 0u;
        uint32_t ci = pieces, li = pieces ? 1u : 0u;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(kFullMask, ci, o), y = __shfl_up_sync(kFullMask, li, o);
            if (lane >= (uint32_t)o) { ci += x; li += y; }
        }
        if (lane == 31) { warp_chunks[warp] = ci; warp_longs[warp] = li; }
        __syncthreads();
        uint32_t c0 = ck, l0 = lr, ct = 0, lt = 0;
        for (uint32_t w = 0; w < kListThreads / 32; ++w) {
            if (w < warp) { c0 += warp_chunks[w]; l0 += warp_longs[w]; }
            ct += warp_chunks[w];
            lt += warp_longs[w];
        }
        if (pieces) {
            const uint32_t q0 = v.rp[r], q1 = v.rp[r + 1], piece = piece_length(sizes, q1 - q0), slot = c0 + ci - pieces, row = l0 + li - 1;
            a.long_rows[row] = LongRow{first + r, slot, slot + pieces, 0u};
            for (uint32_t k = 0; k < pieces; ++k) {
                a.chunks[slot + k] = Chunk{first + r, q0 + k * piece, min(q0 + k * piece + piece, q1), slot + k};
                a.owners[slot + k] = row;
            }
        }
        ck += ct;
        lr += lt;
        __syncthreads();
    }
    const uint32_t t0 = group.y + a.path_tiles[(size_t)seg * kEntries + group.x];
    for (uint32_t k = tid; k < num_starts; k += kListThreads) {
        const uint32_t r = starts[k], e = v.next[r];
        a.tiles[t0 + k] = Tile{first + r, first + e, v.rp[r], v.rp[e]};
    }
    ptx::grid_wait();
}

// ---- panel census: which panels the tensor-core kernel takes ------------------------------------------------------
// Distinct columns of a panel, counted with a hash set in shared memory (open addressing; a 16-row panel holds a few
// hundred nonzeros, so the set is a few KB and a count costs one shared atomic per nonzero, where sorting the panel
// costs 36-91 passes over it: 590 us for R-MAT 2^17 with 1.9 M nonzeros).  A panel is a chain of five latencies, so a
// warp takes one on its own (four at a time per block; a block per panel took 35 us there, with 7 blocks per SM by their
// shared memory); panels of more than kWarpPanelNnz are left to the whole block.  Runs on row pointers nobody
// has checked yet: every position is clamped to nnz = row_ptr[M], and the host drops the result when the check fails.
constexpr int kCensusThreads = 128;
constexpr uint32_t kCensusWarps = kCensusThreads / 32;
constexpr uint32_t kWarpPanelNnz = 512;  // panels up to this are a warp's: four batches of loads

// Inserts the columns col_at(0 .. n-1) into `table` (size a power of two > n, clear): `threads` threads, of which this
// is number `me`; emit(slot) for every slot a new column lands in.
template <class ColAt, class Emit>
__device__ __forceinline__ void hash_insert(uint32_t *table, uint32_t size, uint32_t n, uint32_t me, uint32_t threads, ColAt col_at, Emit emit)
{
    const uint32_t shift = 1 + __clz(size);  // the product's top bits: its low ones see only the column's low bits
    constexpr uint32_t kAhead = 4;  // columns loaded together: the inserts do not wait for one load each
    for (uint32_t i = me; i < n; i += threads * kAhead) {
        uint32_t c[kAhead];
#pragma unroll
        for (uint32_t u = 0; u < kAhead; ++u) c[u] = i + u * threads < n ? col_at(i + u * threads) : 0u;
#pragma unroll
        for (uint32_t u = 0; u < kAhead; ++u) {
            if (i + u * threads >= n) break;
            uint32_t h = (c[u] * 2654435761u) >> shift;
            for (;;) {
                const uint32_t old = atomicCAS(&table[h], 0xffffffffu, c[u]);  // 0xffffffff is no column: K < 2^32
                if (old == 0xffffffffu) { emit(h); break; }
                if (old == c[u]) break;
                h = (h + 1) & (size - 1);
            }
        }
    }
}
// entries of a set for n columns: half full, or up to three quarters where `most` entries are there
__host__ __device__ __forceinline__ uint32_t hash_size(uint32_t n, uint32_t most)
{
    uint32_t size = 64;
    while (size < 2 * n && size < most) size <<= 1;
    return size;
}

// What the census decides about panel q with n nonzeros and nc distinct columns; one thread.
__device__ __forceinline__ void census_result(const CensusArgs &a, uint32_t q, uint32_t n, uint32_t nc, bool candidate)
{
    const uint32_t r0 = q * kPanelRows, r1 = min(a.M, r0 + kPanelRows), padded = (nc + kBrickCols - 1) / kBrickCols * kBrickCols;
    // fill of the panel's 16 x padded dense image, the expression of choose_panel_paths (plan.cpp)
    const bool brick = candidate && (a.force || (float)n / (float)(kPanelRows * padded) >= a.density);
    a.ncols[q] = nc;
    a.path[q] = brick ? 1 : 0;
    if (!brick) return;
    const uint32_t nb = padded / kBrickCols;
    atomicAdd(&a.seg_panels[r0 / kTileSegmentRows], 1u);
    atomicAdd(&a.seg_slots[r0 / kTileSegmentRows], (nb + 3) / 4 * 4);
    atomicAdd(&a.totals->bricks, (unsigned long long)nb);
    atomicAdd(&a.totals->brick_cost, (unsigned long long)n + (r1 - r0) * kRowCost);
    atomicMax(&a.totals->brick_nnz_max, n);
    atomicMax(&a.totals->brick_cols_max, nc);
}

__global__ void __launch_bounds__(kCensusThreads) panel_census_kernel(const uint32_t *__restrict__ row_ptr, const uint32_t *__restrict__ cols, CensusArgs a)
{
    ptx::grid_release();
    extern __shared__ uint32_t table[];
    __shared__ uint32_t distinct, big[kCensusWarps];
    const uint32_t nnz = __ldg(row_ptr + a.M), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t quarter = a.table_words / kCensusWarps;
    uint32_t *mine = table + warp * quarter;
    for (uint32_t q0 = blockIdx.x * kCensusWarps; q0 < a.num_panels; q0 += gridDim.x * kCensusWarps) {
        const uint32_t q = q0 + warp, r0 = q * kPanelRows;
        bool large = false;
        if (q < a.num_panels) {  // uniform across the warp
            const uint32_t r1 = min(a.M, r0 + kPanelRows);
            const uint32_t p = __ldg(row_ptr + min(r0 + lane, r1)), p_next = __shfl_down_sync(kFullMask, p, 1);
            const uint32_t longest = __reduce_max_sync(kFullMask, lane < r1 - r0 && p_next > p ? p_next - p : 0u);
            const uint32_t j0 = min(__shfl_sync(kFullMask, p, 0), nnz), j1 = min(max(__shfl_sync(kFullMask, p, (int)(r1 - r0)), j0), nnz), n = j1 - j0;
            const bool candidate = n != 0 && n <= a.most && (a.force || longest <= a.split_nnz);
            if (n > a.most && lane == 0) atomicAdd(&a.totals->too_large, 1u);
            const uint32_t size = hash_size(n, quarter);
            large = candidate && n > kWarpPanelNnz;
            if (!large) {
                uint32_t got = 0;
                if (candidate) {
                    for (uint32_t i = lane; i < size; i += 32) mine[i] = 0xffffffffu;
                    __syncwarp();
                    hash_insert(mine, size, n, lane, 32, [&](uint32_t i) { return __ldg(cols + j0 + i); }, [&](uint32_t) { ++got; });
                }
                got = __reduce_add_sync(kFullMask, got);
                if (lane == 0) census_result(a, q, n, got, candidate);
                __syncwarp();
            }
        }
        if (lane == 0) big[warp] = large;
        __syncthreads();
        for (uint32_t w = 0; w < kCensusWarps; ++w) {
            if (!big[w]) continue;  // uniform across the block
            const uint32_t qq = q0 + w, j0 = min(__ldg(row_ptr + qq * kPanelRows), nnz),
                           j1 = min(max(__ldg(row_ptr + min(a.M, qq * kPanelRows + kPanelRows)), j0), nnz), n = j1 - j0, size = hash_size(n, a.table_words);
            if (tid == 0) distinct = 0;
            for (uint32_t i = tid; i < size; i += kCensusThreads) table[i] = 0xffffffffu;
            __syncthreads();
            uint32_t got = 0;
            hash_insert(table, size, n, tid, kCensusThreads, [&](uint32_t i) { return __ldg(cols + j0 + i); }, [&](uint32_t) { ++got; });
            got = __reduce_add_sync(kFullMask, got);
            if (lane == 0 && got) atomicAdd(&distinct, got);
            __syncthreads();
            if (tid == 0) census_result(a, qq, n, distinct, true);
            __syncthreads();
        }
        __syncthreads();
    }
    ptx::grid_wait();  // what follows waits for this kernel, and through it for the lists
}

// ---- what the whole matrix looks like --------------------------------------------------------------------------------
// A thread per row.  (1) The nonzeros in rows longer than kDefaultSplitNnz, which item_sizes decides by, and in those that make a
// matrix uneven (mid_row), and the rows that have any.  (2) Whether rows come in runs of the same columns (find_row_runs, plan.cpp): a row is compared with the row in
// front; what is ruled out already is not looked at again, which for most matrices is everything after each block's first
// rows, so the grid is one block per SM at most and a warp reports once.  Positions are clamped to nnz (nobody has checked
// the row pointers yet).  cols may be missing: no runs are looked for then.
__global__ void __launch_bounds__(1024) row_survey_kernel(const uint32_t *__restrict__ row_ptr, const uint32_t *__restrict__ cols, uint32_t M, BuildTotals *totals)
{
    ptx::grid_wait();
    ptx::grid_release();
    volatile uint32_t *unlike = &totals->unlike;
    const uint32_t nnz = __ldg(row_ptr + M), lane = threadIdx.x & 31;
    const uint32_t never = (M % 2 ? 1u : 0u) | (M % 3 ? 2u : 0u);
    uint32_t in_long = 0, in_mid = 0, filled = 0;
    for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); b < M; b += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t known = cols ? __shfl_sync(kFullMask, *unlike | never, 0) : 3u;
        const uint64_t r = b + lane;
        const uint32_t asks = r < M ? ((r % 2 ? 1u : 0u) | (r % 3 ? 2u : 0u)) & ~known : 0u;
        const uint32_t j = min(__ldg(row_ptr + min(r, (uint64_t)M)), nnz), e = min(__ldg(row_ptr + min(r + 1, (uint64_t)M)), nnz);
        const uint32_t len = e > j ? e - j : 0u;
        filled += r < M && len != 0;
        if (len > kDefaultSplitNnz) in_long += len;
        else if (mid_row(len, nnz, M)) in_mid += len;
        uint32_t found = 0;
        if (asks) {
            const uint32_t i = min(__ldg(row_ptr + r - 1), nnz);
            bool same = i <= j && j <= e && j - i == e - j;
            for (uint32_t k = 0; same && j + k < e; ++k) same = __ldg(cols + i + k) == __ldg(cols + j + k);
            if (!same) found = asks;
        }
        found = __reduce_or_sync(kFullMask, found);
        if (found && lane == 0) atomicOr(&totals->unlike, found);
    }
    __shared__ uint32_t warps[3][32];
    in_long = __reduce_add_sync(kFullMask, in_long);
    in_mid = __reduce_add_sync(kFullMask, in_mid);
    filled = __reduce_add_sync(kFullMask, filled);
    if (lane == 0) {
        warps[0][threadIdx.x >> 5] = in_long;
        warps[1][threadIdx.x >> 5] = in_mid;
        warps[2][threadIdx.x >> 5] = filled;
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    in_long = __reduce_add_sync(kFullMask, warps[0][lane]);
    in_mid = __reduce_add_sync(kFullMask, warps[1][lane]);
    filled = __reduce_add_sync(kFullMask, warps[2][lane]);
    if (lane == 0) {
        if (filled) atomicAdd(&totals->filled_rows, filled);
        if (in_long) atomicAdd(&totals->long_nnz, (unsigned long long)in_long);
        if (in_mid) atomicAdd(&totals->mid_nnz, (unsigned long long)in_mid);
    }
}

// ---- slots of the brick stream ------------------------------------------------------------------------------------
// One warp per segment of kTileSegmentRows rows: its panels' slot ranges, from the segment's offsets (lists_scan_kernel).
__global__ void __launch_bounds__(128) brick_layout_kernel(uint32_t num_panels, const uint8_t *__restrict__ path, const uint32_t *__restrict__ ncols,
                                                           const uint32_t *__restrict__ seg_panels, const uint32_t *__restrict__ seg_slots,
                                                           uint32_t num_segments, uint32_t *__restrict__ ids, uint32_t *__restrict__ first,
                                                           uint32_t *__restrict__ last)
{
    ptx::grid_wait();
    ptx::grid_release();
    constexpr uint32_t kPanels = kTileSegmentRows / kPanelRows;
    const uint32_t lane = threadIdx.x & 31, seg = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (seg >= num_segments) return;
    uint32_t at = __ldg(seg_panels + seg), slot = __ldg(seg_slots + seg);
    for (uint32_t b = 0; b < kPanels; b += 32) {
        const uint32_t q = seg * kPanels + b + lane;
        const bool brick = q < num_panels && __ldg(path + q);
        const uint32_t nb = brick ? (__ldg(ncols + q) + kBrickCols - 1) / kBrickCols : 0u, ns = (nb + 3) / 4 * 4;
        uint32_t incl = ns;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= (uint32_t)o) incl += v;
        }
        const unsigned m = __ballot_sync(kFullMask, brick);
        if (brick) {
            const uint32_t i = at + __popc(m & ((1u << lane) - 1u));
            ids[i] = q;
            first[i] = slot + incl - ns;
            last[i] = slot + incl - ns + nb;
        }
        at += __popc(m);
        slot += __shfl_sync(kFullMask, incl, 31);
    }
}

// position of (row r, column c) of a 16 x 8 brick in its record, in mma.m16n8k8 A-fragment order (plan.hpp)
__device__ __forceinline__ uint32_t frag_index(uint32_t r, uint32_t c) { return ((r & 7u) * 4u + (c & 3u)) * 4u + (r >> 3) + 2u * (c >> 2); }

// ---- brick records of the panels routed to the tensor-core kernel ----------------------------------------------
// One block per brick panel: the distinct columns (hash set, then a bitonic sort of the distinct ones only), the
// panel's column list (8 per slot) and records; then every thread drops nonzeros into their bricks.  A position named
// twice must add up in storage order, as in the host builder: when a thread meets a position that is already taken, the
// panel is written once more, one thread per row in storage order.
__global__ void __launch_bounds__(kCensusThreads) brick_fill_kernel(const uint32_t *__restrict__ row_ptr, const uint2 *__restrict__ pairs, uint32_t M,
                                                                    const uint32_t *__restrict__ ids, const uint32_t *__restrict__ first_slot,
                                                                    uint32_t num_brick_panels, const uint32_t *__restrict__ ncols, uint32_t table_words,
                                                                    uint32_t list_words, uint32_t *__restrict__ bcols, uint32_t *__restrict__ brecs)
{
    ptx::grid_wait();
    ptx::grid_release();
    extern __shared__ uint32_t table[];
    uint32_t *list = table + table_words;   // the panel's distinct columns, ascending
    uint32_t *map = list + list_words;      // occupancy: 4 words per brick
    __shared__ uint32_t count, twice;
    const uint32_t tid = threadIdx.x;
    for (uint32_t i = blockIdx.x; i < num_brick_panels; i += gridDim.x) {
        const uint32_t q = __ldg(ids + i), nc = __ldg(ncols + q), f = __ldg(first_slot + i);
        const uint32_t r0 = q * kPanelRows, r1 = min(M, r0 + kPanelRows), j0 = __ldg(row_ptr + r0), n = __ldg(row_ptr + r1) - j0;
        const uint32_t nb = (nc + kBrickCols - 1) / kBrickCols, nslots = (nb + 3) / 4 * 4;
        const uint32_t size = hash_size(n, table_words);
        uint32_t sorted = 1;
        while (sorted < nc) sorted <<= 1;
        if (tid == 0) count = twice = 0;
        for (uint32_t k = tid; k < size; k += kCensusThreads) table[k] = 0xffffffffu;
        for (uint32_t k = tid; k < sorted; k += kCensusThreads) list[k] = 0xffffffffu;
        for (uint32_t k = tid; k < nb * 4; k += kCensusThreads) map[k] = 0u;
        uint4 *rec4 = reinterpret_cast<uint4 *>(brecs + (size_t)f * kBrickRecWords);
        for (uint32_t k = tid; k < nslots * (kBrickRecWords / 4); k += kCensusThreads) rec4[k] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        hash_insert(table, size, n, tid, kCensusThreads, [&](uint32_t k) { return __ldg(&pairs[j0 + k].x); }, [&](uint32_t h) { list[atomicAdd(&count, 1u)] = table[h]; });
        __syncthreads();
        for (uint32_t k = 2; k <= sorted; k <<= 1)
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                for (uint32_t x = tid; x < sorted; x += kCensusThreads) {
                    const uint32_t y = x ^ j;
                    if (y > x) {
                        const uint32_t u = list[x], v = list[y];
                        if ((u > v) == ((x & k) == 0)) {
                            list[x] = v;
                            list[y] = u;
                        }
                    }
                }
                __syncthreads();
            }
        for (uint32_t c = tid; c < nslots * kBrickCols; c += kCensusThreads) bcols[(size_t)f * kBrickCols + c] = list[min(c, nc - 1)];
        auto place = [&](uint32_t row, uint32_t j, bool in_order) {
            const uint2 pr = __ldg(pairs + j);
            uint32_t lo = 0, hi = nc;  // first position with list[pos] >= column (the column is in the list)
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (list[mid] < pr.x) lo = mid + 1; else hi = mid;
            }
            const uint32_t b = lo / kBrickCols, bit = row * kBrickCols + lo % kBrickCols;
            const bool taken = (atomicOr(&map[b * 4 + (bit >> 5)], 1u << (bit & 31)) >> (bit & 31)) & 1u;
            float *at = reinterpret_cast<float *>(brecs + (size_t)(f + b) * kBrickRecWords + kBrickRecHeaderWords + frag_index(row, lo % kBrickCols));
            const float v = __uint_as_float(pr.y);
            if (taken && !in_order) twice = 1;
            *at = taken && in_order ? *at + v : v;
        };
        for (uint32_t r = r0 + (tid >> 3); r < r1; r += kCensusThreads / 8)  // eight threads per row
            for (uint32_t j = __ldg(row_ptr + r) + (tid & 7), je = __ldg(row_ptr + r + 1); j < je; j += 8) place(r - r0, j, false);
        __syncthreads();
        if (twice) {  // uniform
            for (uint32_t k = tid; k < nb * 4; k += kCensusThreads) map[k] = 0u;
            __syncthreads();
            if (r0 + tid < r1)
                for (uint32_t j = __ldg(row_ptr + r0 + tid), je = __ldg(row_ptr + r0 + tid + 1); j < je; ++j) place(tid, j, true);
            __syncthreads();
        }
        for (uint32_t b = tid; b < nb; b += kCensusThreads) {
            uint32_t *rec = brecs + (size_t)(f + b) * kBrickRecWords;
            for (int w = 0; w < 4; ++w) rec[w] = map[b * 4 + w];
            rec[4] = b + 1 == nb ? 1u : 0u;
            rec[5] = q;
        }
        __syncthreads();
    }
}

// The plan's own arrays from the caller's CSR in one pass: (column, value) pairs with the column range checked, the row
// pointers, and the slack behind both that the tile copies may read.  Bound by memory: 16 bytes per nonzero.
__global__ void __launch_bounds__(256) pack_kernel(const uint32_t *__restrict__ row_ptr, const uint32_t *__restrict__ cols, const float *__restrict__ vals,
                                                   uint32_t M, uint32_t K, uint32_t nnz, uint32_t *__restrict__ row_ptr_out, uint2 *__restrict__ pairs,
                                                   uint32_t *__restrict__ bad)
{
    ptx::grid_release();
    ptx::grid_wait();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool out_of_range = false;
    for (uint64_t j = t0; j < (uint64_t)nnz + 2; j += stride) {
        uint2 pr = make_uint2(0u, 0u);
        if (j < nnz) {
            pr = make_uint2(__ldcs(cols + j), __float_as_uint(__ldcs(vals + j)));
            out_of_range |= pr.x >= K;
        }
        pairs[j] = pr;
    }
    for (uint64_t r = t0; r < (uint64_t)M + 1 + kRowPtrSlack; r += stride) row_ptr_out[r] = __ldg(row_ptr + (r < M ? r : M));
    if (__any_sync(kFullMask, out_of_range) && (threadIdx.x & 31) == 0) atomicOr(bad, 1u);
}

// pairs[j].value = vals[order[j]] (order may be absent): new values for an unchanged pattern.
template <bool ORDER>
__global__ void __launch_bounds__(256) set_values_kernel(uint2 *__restrict__ pairs, const float *__restrict__ vals, const uint32_t *__restrict__ order,
                                                         uint64_t nnz)
{
    ptx::grid_wait();
    ptx::grid_release();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < nnz; j += stride)
        pairs[j].y = __float_as_uint(ORDER ? __ldg(vals + __ldcs(order + j)) : __ldcs(vals + j));
}

__global__ void __launch_bounds__(256) unpack_kernel(const uint2 *__restrict__ pairs, uint32_t *__restrict__ cols, float *__restrict__ vals, uint64_t nnz)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < nnz; j += stride) {
        const uint2 pr = __ldcs(pairs + j);
        cols[j] = pr.x;
        if (vals) vals[j] = __uint_as_float(pr.y);
    }
}

}  // namespace

cudaError_t launch_set_values(void *pairs, const float *vals, const uint32_t *order, uint64_t nnz, int sm_count, cudaStream_t s)
{
    if (nnz == 0) return cudaSuccess;
    const uint32_t blocks = (uint32_t)std::min<uint64_t>((nnz + 255) / 256, (uint64_t)sm_count * 8);
    return launch_overlapped(order ? set_values_kernel<true> : set_values_kernel<false>, blocks, 256, 0, s, static_cast<uint2 *>(pairs), vals, order, nnz);
}

cudaError_t launch_unpack(const void *pairs, uint32_t *cols, float *vals, uint64_t nnz, int sm_count, cudaStream_t s)
{
    if (nnz == 0) return cudaSuccess;
    const uint32_t blocks = (uint32_t)std::min<uint64_t>((nnz + 255) / 256, (uint64_t)sm_count * 8);
    unpack_kernel<<<blocks, 256, 0, s>>>(static_cast<const uint2 *>(pairs), cols, vals, nnz);
    return cudaGetLastError();
}

cudaError_t launch_pack(const uint32_t *row_ptr, const uint32_t *cols, const float *vals, uint32_t M, uint32_t K, uint32_t nnz, uint32_t *row_ptr_out,
                        void *pairs, uint32_t *bad, int sm_count, cudaStream_t s)
{
    const uint64_t items = std::max<uint64_t>((uint64_t)nnz + 2, (uint64_t)M + 1 + kRowPtrSlack);
    const uint32_t blocks = (uint32_t)std::min<uint64_t>((items + 255) / 256, (uint64_t)sm_count * 8);
    return launch_overlapped(pack_kernel, blocks, 256, 0, s, row_ptr, cols, vals, M, K, nnz, row_ptr_out, static_cast<uint2 *>(pairs), bad);
}

cudaError_t launch_lists_count(const uint32_t *row_ptr, const ListArgs &a, cudaStream_t s)
{
    if (a.num_segments == 0) return cudaSuccess;
    return launch_overlapped(lists_count_kernel, a.num_segments, kListThreads, 0, s, row_ptr, a);
}

cudaError_t launch_lists_scan(const uint32_t *row_ptr, const ListArgs &a, uint32_t *counters, uint32_t how_many, cudaStream_t s)
{
    if (a.num_segments) {
        const cudaError_t e = launch_overlapped(lists_compose_kernel, (a.num_segments + kGroup - 1) / kGroup, kListThreads, 0, s, a);
        if (e != cudaSuccess) return e;
    }
    return launch_overlapped(lists_scan_kernel, 1 + how_many, 1024, 0, s, row_ptr, a, counters);
}

cudaError_t launch_lists_write(const uint32_t *row_ptr, const ListArgs &a, cudaStream_t s)
{
    if (a.num_segments == 0) return cudaSuccess;
    return launch_overlapped(lists_write_kernel, a.num_segments, kListThreads, 0, s, row_ptr, a);
}

cudaError_t launch_panel_census(const uint32_t *row_ptr, const uint32_t *cols, CensusArgs a, int sm_count, cudaStream_t s)
{
    if (a.num_panels == 0) return cudaSuccess;
    // a hash set at most three quarters full: kMaxCensusNnz nonzeros (auto: 16 rows that are not long) or kDevPanelMax
    a.most = a.force ? kDevPanelMax : kMaxCensusNnz;
    a.table_words = a.force ? 16384 : 8192;
    const int smem = (int)a.table_words * 4;
    cudaError_t e = allow_dynamic_smem<panel_census_kernel>(16384 * 4);
    if (e != cudaSuccess) return e;
    const uint32_t blocks = std::min((a.num_panels + kCensusWarps - 1) / kCensusWarps, (uint32_t)sm_count * 16);
    return launch_overlapped(panel_census_kernel, blocks, kCensusThreads, smem, s, row_ptr, cols, a);
}

cudaError_t launch_row_survey(const uint32_t *row_ptr, const uint32_t *cols, uint32_t M, BuildTotals *totals, int sm_count, cudaStream_t s)
{
    if (M == 0) return cudaSuccess;
    return launch_overlapped(row_survey_kernel, std::min((M + 1023) / 1024, (uint32_t)sm_count), 1024, 0, s, row_ptr, cols, M, totals);
}

cudaError_t launch_brick_layout(uint32_t num_panels, const uint8_t *path, const uint32_t *ncols, const uint32_t *seg_panels, const uint32_t *seg_slots,
                                uint32_t num_segments, uint32_t *ids, uint32_t *first, uint32_t *last, cudaStream_t s)
{
    return launch_overlapped(brick_layout_kernel, (num_segments + 3) / 4, 128, 0, s, num_panels, path, ncols, seg_panels, seg_slots, num_segments, ids, first, last);
}

cudaError_t launch_panel_columns(const uint32_t *row_ptr, const void *pairs, uint32_t M, uint32_t num_panels, uint32_t *ncols,
                                 uint32_t *acols, int sm_count, cudaStream_t s)
{
    if (num_panels == 0) return cudaSuccess;
    const uint32_t blocks = num_panels < (uint32_t)sm_count * 16 ? num_panels : (uint32_t)sm_count * 16;
    panel_columns_kernel<<<blocks, 256, kDevPanelMax * sizeof(uint32_t), s>>>(row_ptr, static_cast<const uint2 *>(pairs), M, num_panels,
                                                                              ncols, acols);
    return cudaGetLastError();
}

cudaError_t launch_panel_max_col(const uint32_t *row_ptr, const void *pairs, uint32_t M, uint32_t num_panels, uint32_t *maxcol, int sm_count,
                                 cudaStream_t s)
{
    if (num_panels == 0) return cudaSuccess;
    const uint32_t want = (num_panels + 7) / 8;
    const uint32_t blocks = want < (uint32_t)sm_count * 8 ? want : (uint32_t)sm_count * 8;
    panel_max_col_kernel<<<blocks, 256, 0, s>>>(row_ptr, static_cast<const uint2 *>(pairs), M, num_panels, maxcol);
    return cudaGetLastError();
}

cudaError_t launch_brick_fill(const uint32_t *row_ptr, const void *pairs, uint32_t M, const uint32_t *ids, const uint32_t *first_slot,
                              uint32_t num_brick_panels, const uint32_t *ncols, uint32_t nnz_max, uint32_t cols_max, uint32_t *bcols, uint32_t *brecs,
                              int sm_count, cudaStream_t s)
{
    if (num_brick_panels == 0) return cudaSuccess;
    uint32_t table = hash_size(nnz_max, 16384), list = 1;
    while (list < cols_max) list <<= 1;
    list = (list + 3) / 4 * 4;
    const uint32_t map = (cols_max + kBrickCols - 1) / kBrickCols * 4;
    cudaError_t e = allow_dynamic_smem<brick_fill_kernel>((16384 + kDevPanelMax + kDevPanelMax / kBrickCols * 4) * 4);
    if (e != cudaSuccess) return e;
    return launch_overlapped(brick_fill_kernel, std::min(num_brick_panels, (uint32_t)sm_count * 16), kCensusThreads, (table + list + map) * 4, s,
                             row_ptr, static_cast<const uint2 *>(pairs), M, ids, first_slot, num_brick_panels, ncols, table, list, bcols, brecs);
}

}  // namespace cutespmm

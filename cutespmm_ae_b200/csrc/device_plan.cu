// cutespmm_plan_create_device: a plan from CSR arrays that live on the GPU.  The counting kernels run first (row
// pointers checked, work lists and panels counted), one small read tells the host the sizes, one block of memory is taken
// for the whole plan and the writing kernels fill it; a second wait ends the call.  What the host keeps is sizes: the
// lists themselves come to the host only when a caller asks for something that needs them (decode, save, the panel
// views, the host-buffer call in blocks of rows).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "device_plan.hpp"
#include "nvtx.hpp"
#include "plan_object.hpp"

using namespace cutespmm;

namespace {

// ---- memory of device-built plans ----------------------------------------------------------------------------------
// A program whose graph changes from step to step makes and drops a plan per step; cudaMalloc and cudaFree (which waits
// for the whole device) would be most of its time.  So these plans' memory comes from a stream-ordered pool of the
// library's own, one per device, thread-safe in the driver.  The pool keeps at most kPoolKeeps bytes beyond what
// living plans hold across a synchronisation (the rest goes back to the driver), and gives them up when an allocation
// fails or cutespmm_release_memory is called.
constexpr uint64_t kPoolKeeps = 1ull << 30, kPoolStep = 128ull << 20;
constexpr int kMaxDevices = 64;

std::mutex g_device_mutex;
cudaMemPool_t g_pool[kMaxDevices] = {};
uint64_t g_pool_live[kMaxDevices] = {}, g_pool_threshold[kMaxDevices] = {};
int g_sm_count[kMaxDevices] = {};

// Bytes of living plans changed: the driver's threshold counts them too, so it moves along (in steps, to be set rarely).
void note_live(int dev, int64_t change)
{
    std::lock_guard<std::mutex> lock(g_device_mutex);
    g_pool_live[dev] += (uint64_t)change;
    uint64_t want = g_pool_live[dev] / kPoolStep * kPoolStep + kPoolKeeps;
    if (g_pool[dev] && want != g_pool_threshold[dev] && cudaMemPoolSetAttribute(g_pool[dev], cudaMemPoolAttrReleaseThreshold, &want) == cudaSuccess)
        g_pool_threshold[dev] = want;
}

cudaError_t device_pool(int dev, cudaMemPool_t *pool)
{
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_device_mutex);
    if (!g_pool[dev]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaError_t e = cudaMemPoolCreate(&g_pool[dev], &props);
        if (e != cudaSuccess) { g_pool[dev] = nullptr; return e; }
        uint64_t keep = g_pool_threshold[dev] = kPoolKeeps;
        if ((e = cudaMemPoolSetAttribute(g_pool[dev], cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) return e;
    }
    *pool = g_pool[dev];
    return cudaSuccess;
}

// Hands out 256-byte aligned parts of one block.
struct Carver {
    char *base = nullptr;
    uint64_t used = 0;
    template <class T> void take(T *&p, uint64_t count)
    {
        p = reinterpret_cast<T *>(base + used);
        used += (count * sizeof(T) + 255) / 256 * 256;
    }
};

// A pinned slot device words arrive in (a copy to pageable memory costs a staging pass more).
struct Landing {
    uint32_t *slot = nullptr;
    cudaStream_t s;
    explicit Landing(cudaStream_t stream) : s(stream) {}
    ~Landing() { if (slot) cutespmm_internal_give_status_word(slot); }
    template <class T> cudaError_t fetch(T &out, const T *device)  // waits for the stream
    {
        static_assert(sizeof(T) <= kStatusSlotBytes, "one slot");
        cudaError_t e = slot ? cudaSuccess : cutespmm_internal_take_status_word(&slot);
        if (e != cudaSuccess || (e = cudaMemcpyAsync(slot, device, sizeof(T), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return e;
        e = cudaStreamSynchronize(s);
        std::memcpy(&out, slot, sizeof(T));
        return e;
    }
};

struct Temp {  // stream-ordered scratch of one call
    void *p = nullptr;
    cudaStream_t s;
    explicit Temp(cudaStream_t stream) : s(stream) {}
    ~Temp() { if (p) cudaFreeAsync(p, s); }
};

}  // namespace

cudaError_t cutespmm_internal_pool_alloc(void **p, uint64_t bytes, int dev, cudaStream_t s, bool may_wait)
{
    cudaMemPool_t pool = nullptr;
    cudaError_t e = device_pool(dev, &pool);
    if (e != cudaSuccess) return e;
    if ((e = cudaMallocFromPoolAsync(p, bytes, pool, s)) != cudaErrorMemoryAllocation || !may_wait) return e;
    cudaGetLastError();
    cudaStreamSynchronize(s);
    cudaMemPoolTrimTo(pool, 0);
    return cudaMallocFromPoolAsync(p, bytes, pool, s);
}

// The current device, checked to be one this library runs on (the properties are read once per device).
int cutespmm_internal_usable_device(int *dev, int *sm_count)
{
    cudaError_t e = cudaGetDevice(dev);
    if (e != cudaSuccess) return fail_cuda_status(e, "cudaGetDevice (libcutespmm needs a CUDA device; there is no CPU path)");
    const bool cached = *dev >= 0 && *dev < kMaxDevices;
    std::lock_guard<std::mutex> lock(g_device_mutex);
    if (cached && g_sm_count[*dev]) {
        *sm_count = g_sm_count[*dev];
        return CUTESPMM_OK;
    }
    int major = 0, minor = 0;
    if ((e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, *dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, *dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(sm_count, cudaDevAttrMultiProcessorCount, *dev)) != cudaSuccess)
        return fail_cuda_status(e, "cudaDeviceGetAttribute");
    if (major < 10)
        return fail_status(CUTESPMM_EUNSUPPORTED, "this library is built for sm_100a (B200) only; found compute capability " +
                                                      std::to_string(major) + "." + std::to_string(minor));
    if (cached) g_sm_count[*dev] = *sm_count;
    return CUTESPMM_OK;
}

// The block of a device-built plan goes back to the pool.  cudaFree waited for everything on the device; here the block
// is handed back in the order of the default stream, which is enough for a plan that ran on no other (stream handles
// of a caller may be gone by now, so nothing can be recorded on them), and after a wait for the device otherwise.
void cutespmm_internal_free_block(void *block, uint64_t bytes, int dev, bool used_elsewhere)
{
    if (bytes > kPoolKeeps) {
        cudaFree(block);  // not from the pool
        return;
    }
    if (used_elsewhere) cudaDeviceSynchronize();
    if (cudaFreeAsync(block, nullptr) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(block);
    }
    note_live(dev, -(int64_t)bytes);
}

namespace {

int fetch_lists(cutespmm_plan *p)  // p->fetch_mutex held
{
    HostPlan &h = p->host;
    if (p->lists_on_host) return CUTESPMM_OK;
    int cur = -1;
    cudaGetDevice(&cur);
    if (cur != p->device) cudaSetDevice(p->device);
    cudaError_t e = cudaSuccess;
    auto fetch = [&](auto &v, const void *d, uint64_t n) {
        v.resize(n);
        if (n && e == cudaSuccess) e = cudaMemcpy(v.data(), d, n * sizeof(v[0]), cudaMemcpyDeviceToHost);
    };
    int st = CUTESPMM_OK;
    uint32_t *d_max = nullptr;
    try {
        const uint64_t P = h.num_panels();
        fetch(h.row_ptr, p->d_row_ptr, h.M + 1);
        fetch(h.tiles, p->d_tiles, p->own.tiles);
        fetch(h.chunks, p->d_chunks, p->own.chunks);
        fetch(h.long_rows, p->d_long_rows, p->own.long_rows);
        fetch(h.tiles_all, p->d_tiles_all, p->every.tiles);
        fetch(h.chunks_all, p->d_chunks_all, p->every.chunks);
        fetch(h.long_rows_all, p->d_long_rows_all, p->every.long_rows);
        fetch(h.brick_panel_ids, p->d_panel_ids, h.brick_panels);
        fetch(h.panel_first_brick, p->d_panel_first, h.brick_panels);
        fetch(h.panel_last_brick, p->d_panel_last, h.brick_panels);
        h.row_path.assign(P, 0);
        for (uint32_t q : h.brick_panel_ids)
            if (q < P) h.row_path[q] = 1;
        h.slab_path.assign((h.M + kSlabRows - 1) / kSlabRows, 0);
        h.panel_max_col.assign(P, 0u);
        if (P && h.nnz && e == cudaSuccess) {
            if ((e = cudaMalloc(&d_max, P * sizeof(uint32_t))) == cudaSuccess &&
                (e = launch_panel_max_col(static_cast<const uint32_t *>(p->d_row_ptr), p->d_pairs, (uint32_t)h.M, (uint32_t)P, d_max, p->sm_count, nullptr)) == cudaSuccess)
                e = cudaMemcpy(h.panel_max_col.data(), d_max, P * sizeof(uint32_t), cudaMemcpyDeviceToHost);
        }
        if (e != cudaSuccess) st = fail_cuda_status(e, "reading the plan's lists back");
    } catch (const std::bad_alloc &) {
        st = fail_status(CUTESPMM_ENOMEM, "host allocation failed");
    }
    if (d_max) cudaFree(d_max);
    if (cur != p->device && cur >= 0) cudaSetDevice(cur);
    p->lists_on_host = st == CUTESPMM_OK;
    return st;
}

}  // namespace

// The lists of a device-built plan on the host (p->host); nothing to do for a host-built one.
int cutespmm_internal_fetch_lists(const cutespmm_plan *cp)
{
    cutespmm_plan *p = const_cast<cutespmm_plan *>(cp);  // a cache: the plan means the same before and after
    std::lock_guard<std::mutex> lock(p->fetch_mutex);
    return fetch_lists(p);
}

// The panel views of a device-built plan (host.blocked_row_ptr, and the panels' columns when `acols` is given): the panel
// analysis runs now.  Without views (path rows, or a panel beyond the device sort) blocked_row_ptr stays empty.
int cutespmm_internal_fetch_views(const cutespmm_plan *cp, std::vector<uint32_t> *ncols_out, std::vector<uint32_t> *acols_out)
{
    cutespmm_plan *p = const_cast<cutespmm_plan *>(cp);
    std::lock_guard<std::mutex> lock(p->fetch_mutex);
    HostPlan &h = p->host;
    if (!h.device_built || h.opts.path == CUTESPMM_PATH_ROWS || !p->on_device) return CUTESPMM_OK;
    if (p->views_tried && !acols_out) return CUTESPMM_OK;
    const uint64_t P = h.num_panels();
    int cur = -1;
    cudaGetDevice(&cur);
    if (cur != p->device) cudaSetDevice(p->device);
    uint32_t *d_ncols = nullptr, *d_acols = nullptr;
    cudaError_t e = cudaSuccess;
    int st = CUTESPMM_OK;
    try {
        std::vector<uint32_t> ncols(P, 0u);
        if (P && h.nnz) {
            if ((e = cudaMalloc(&d_ncols, P * sizeof(uint32_t))) == cudaSuccess && (e = cudaMalloc(&d_acols, h.nnz * sizeof(uint32_t))) == cudaSuccess &&
                (e = launch_panel_columns(static_cast<const uint32_t *>(p->d_row_ptr), p->d_pairs, (uint32_t)h.M, (uint32_t)P, d_ncols, d_acols, p->sm_count, nullptr)) == cudaSuccess)
                e = cudaMemcpy(ncols.data(), d_ncols, P * sizeof(uint32_t), cudaMemcpyDeviceToHost);
            if (e == cudaSuccess && acols_out) {
                acols_out->resize(h.nnz);
                e = cudaMemcpy(acols_out->data(), d_acols, h.nnz * sizeof(uint32_t), cudaMemcpyDeviceToHost);
            }
        }
        if (e != cudaSuccess) {
            st = fail_cuda_status(e, "panel analysis");
        } else {
            bool complete = true;
            std::vector<uint32_t> brp(P + 1, 0u);
            for (uint64_t q = 0; q < P; ++q) {
                complete &= ncols[q] != kPanelTooLarge;
                brp[q + 1] = brp[q] + (complete ? (ncols[q] + kBlockCols - 1) / kBlockCols : 0);
            }
            if (complete) h.blocked_row_ptr = std::move(brp);
            else h.blocked_row_ptr.clear();
            p->views_tried = true;
            if (ncols_out) *ncols_out = std::move(ncols);
        }
    } catch (const std::bad_alloc &) {
        st = fail_status(CUTESPMM_ENOMEM, "host allocation failed");
    }
    if (d_ncols) cudaFree(d_ncols);
    if (d_acols) cudaFree(d_acols);
    if (cur != p->device && cur >= 0) cudaSetDevice(cur);
    return st;
}

extern "C" {

int cutespmm_release_memory(void)
{
    std::lock_guard<std::mutex> lock(g_device_mutex);
    for (cudaMemPool_t pool : g_pool)
        if (pool) {
            const cudaError_t e = cudaMemPoolTrimTo(pool, 0);
            if (e != cudaSuccess) return fail_cuda_status(e, "cudaMemPoolTrimTo");
        }
    return CUTESPMM_OK;
}

int cutespmm_plan_create_device(cutespmm_plan_t **plan, uint64_t M64, uint64_t K64, const uint32_t *rowPtr_dev, const uint32_t *cols_dev,
                                const float *vals_dev, const cutespmm_options_t *opts, void *stream)
{
    if (!plan) return fail_status(CUTESPMM_EINVAL, "plan is NULL");
    *plan = nullptr;
    if (!rowPtr_dev) return fail_status(CUTESPMM_EINVAL, "rowPtr is NULL");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    NvtxRange range("cutespmm: plan creation (device CSR)");
    int dev = -1, sms = 0;
    int st = cutespmm_internal_usable_device(&dev, &sms);
    if (st != CUTESPMM_OK) return st;
    if (dev >= kMaxDevices) return fail_status(CUTESPMM_EUNSUPPORTED, "device ordinal too large");
    struct Owner {  // drops the plan on every early return
        cutespmm_plan *p = new (std::nothrow) cutespmm_plan();
        ~Owner() { delete p; }
    } owner;
    cutespmm_plan *p = owner.p;
    if (!p) return fail_status(CUTESPMM_ENOMEM, "host allocation failed");
    HostPlan &h = p->host;
    std::string err;
    if ((st = check_device_options(h, M64, K64, opts, err)) != CUTESPMM_OK) return fail_status(st, err);
    p->device = dev;
    p->sm_count = sms;
    p->on_device = true;
    p->lists_on_host = false;
    p->used_elsewhere = true;  // until the call has waited for its own kernels
    const uint32_t M = (uint32_t)M64, K = (uint32_t)K64, P = (uint32_t)h.num_panels();
    const uint32_t segments = (uint32_t)((M64 + kTileSegmentRows - 1) / kTileSegmentRows);
    // path auto puts a panel on the tensor cores only where min_brick_panels of them qualify: fewer panels need no census
    const bool brick_path = h.opts.path == CUTESPMM_PATH_BRICK;
    const bool census = brick_path || (h.opts.path == CUTESPMM_PATH_AUTO && P >= h.opts.min_brick_panels);

    // ---- count ----
    cudaError_t e;
    Temp temp(s);
    BuildTotals *d_totals = nullptr, *d_totals2 = nullptr;
    uint32_t *counters = nullptr, *counters2 = nullptr, *path_tiles = nullptr, *group_tiles = nullptr, *ncols = nullptr;
    uint2 *group_entry = nullptr;
    uint16_t *tables = nullptr, *path_entry = nullptr, *group_exit = nullptr;
    uint8_t *path = nullptr;
    auto carve_temp = [&](Carver &c) {
        c.take(d_totals, 1);
        c.take(d_totals2, 1);
        c.take(counters, 4ull * segments);  // chunks, long rows, brick panels, brick slots
        const uint64_t zeroed = c.used;
        c.take(counters2, census ? 2ull * segments : 0);
        // the tables of both lists (the second only where there may be one)
        const uint64_t lists = census ? 2 : 1, entries = lists * segments * kSegmentEntries, groups = lists * (segments / 32 + 1);
        c.take(tables, 2 * entries);
        c.take(path_entry, entries);
        c.take(path_tiles, entries);
        c.take(group_exit, groups * kSegmentEntries);
        c.take(group_tiles, groups * kSegmentEntries);
        c.take(group_entry, groups);
        c.take(ncols, census ? P : 0);
        c.take(path, census ? P : 0);
        return zeroed;
    };
    Carver sizes;
    carve_temp(sizes);
    if ((e = cutespmm_internal_pool_alloc(&temp.p, sizes.used, dev, s, true)) != cudaSuccess) return fail_cuda_status(e, "scratch of the plan creation");
    Carver at;
    at.base = static_cast<char *>(temp.p);
    const uint64_t zeroed = carve_temp(at);
    ListArgs la{};
    la.M = M; la.num_segments = segments;
    la.split_nnz = h.opts.split_nnz; la.tile_nnz = h.opts.tile_nnz; la.adaptive = h.adaptive_tiling ? 1u : 0u;
    auto set_tables = [&](ListArgs &l, uint64_t list) {
        const uint64_t entries = (uint64_t)segments * kSegmentEntries, groups = segments / 32 + 1;
        l.exits = tables + 2 * list * entries; l.tile_counts = l.exits + entries;
        l.path_entry = path_entry + list * entries; l.path_tiles = path_tiles + list * entries;
        l.group_exit = group_exit + list * groups * kSegmentEntries; l.group_tiles = group_tiles + list * groups * kSegmentEntries;
        l.group_entry = group_entry + list * groups;
    };
    set_tables(la, 0);
    la.seg_chunks = counters; la.seg_longs = counters + segments;
    la.totals = d_totals;
    la.long_nnz = &d_totals->long_nnz;
    CensusArgs ca{};
    ca.M = M; ca.num_panels = P; ca.force = brick_path ? 1u : 0u;
    ca.split_nnz = h.opts.split_nnz; ca.density = h.opts.brick_density;
    ca.ncols = ncols; ca.path = path;
    ca.seg_panels = counters + 2ull * segments; ca.seg_slots = counters + 3ull * segments;
    ca.totals = d_totals;
    Landing landing(s);
    BuildTotals t{};
    if ((e = cudaMemsetAsync(temp.p, 0, zeroed, s)) != cudaSuccess || (e = launch_row_survey(rowPtr_dev, cols_dev, M, d_totals, sms, s)) != cudaSuccess ||
        (e = launch_lists_count(rowPtr_dev, la, s)) != cudaSuccess ||
        (census && cols_dev && (e = launch_panel_census(rowPtr_dev, cols_dev, ca, sms, s)) != cudaSuccess) ||
        (e = launch_lists_scan(rowPtr_dev, la, counters, census ? 4 : 2, s)) != cudaSuccess ||
        (e = landing.fetch(t, d_totals)) != cudaSuccess)
        return fail_cuda_status(e, "reading the row pointers");
    h.nnz = t.nnz;
    h.uneven = is_uneven(t.mid_nnz, t.long_nnz, t.nnz);
    h.filled_rows = t.filled_rows;
    h.run_rows = M < 2 || !t.nnz ? 0 : M % 3 == 0 && !(t.unlike & 2) ? 3 : M % 2 == 0 && !(t.unlike & 1) ? 2 : 0;
    if (t.bad_rows || (M == 0 && t.nnz)) return fail_status(CUTESPMM_EINVAL, "rowPtr must start at 0 and be non-decreasing");
    if (h.nnz && (!cols_dev || !vals_dev)) return fail_status(CUTESPMM_EINVAL, "cols/vals is NULL");
    if (brick_path && t.too_large)
        return fail_status(CUTESPMM_EUNSUPPORTED, "path brick on the device: a 16-row panel holds more than " + std::to_string(kDevPanelMax) +
                                                      " nonzeros; use path auto (such panels run on the row kernel) or the host builder");
    const bool bricks = census && t.brick_panels && (brick_path || t.brick_panels >= h.opts.min_brick_panels);
    p->own = {t.tiles, t.chunks, t.long_rows};
    ListArgs la2 = la;
    if (bricks) {  // two lists: every row, and the rows the bricks leave
        p->every = p->own;
        h.brick_panels = t.brick_panels;
        h.num_bricks = t.bricks;
        h.brick_slots = t.brick_slots;
        la2.path = path;
        la2.total_known = 1;
        la2.total = h.nnz + (uint64_t)kRowCost * M - t.brick_cost;
        set_tables(la2, 1);
        la2.seg_chunks = counters2; la2.seg_longs = counters2 + segments;
        la2.totals = d_totals2;
        BuildTotals t2{};
        if ((e = launch_lists_count(rowPtr_dev, la2, s)) != cudaSuccess ||
            (e = launch_lists_scan(rowPtr_dev, la2, counters2, 2, s)) != cudaSuccess ||
            (e = landing.fetch(t2, d_totals2)) != cudaSuccess)
            return fail_cuda_status(e, "counting the work lists");
        p->own = {t2.tiles, t2.chunks, t2.long_rows};
    }

    // ---- one block for everything ----
    const uint64_t col_words = h.brick_slots * kBrickCols + 96, rec_words = h.brick_slots * kBrickRecWords;
    const uint64_t slots = std::max(p->own.chunks, p->every.chunks), longs = (uint64_t)p->own.long_rows + p->every.long_rows;
    uint32_t *d_rp = nullptr, *d_owner = nullptr, *d_owner_all = nullptr, *d_bcols = nullptr, *d_brecs = nullptr, *d_first = nullptr, *d_last = nullptr, *d_ids = nullptr;
    Pair *d_pairs = nullptr;
    Tile *d_tiles = nullptr, *d_tiles_all = nullptr;
    Chunk *d_chunks = nullptr, *d_chunks_all = nullptr;
    LongRow *d_longs = nullptr, *d_longs_all = nullptr;
    auto carve = [&](Carver &c) {
        c.take(p->d_status, 64);
        c.take(p->d_arrivals, longs * kArrivalStride);
        const uint64_t zero = c.used;
        c.take(d_rp, (uint64_t)M + 1 + kRowPtrSlack);
        c.take(d_pairs, h.nnz + 2);
        c.take(d_tiles, p->own.tiles);
        c.take(d_chunks, p->own.chunks);
        c.take(d_longs, p->own.long_rows);
        c.take(d_owner, p->own.chunks);
        c.take(d_tiles_all, p->every.tiles);
        c.take(d_chunks_all, p->every.chunks);
        c.take(d_longs_all, p->every.long_rows);
        c.take(d_owner_all, p->every.chunks);
        if (bricks) {
            c.take(d_bcols, col_words);
            c.take(d_brecs, rec_words);
            c.take(d_first, h.brick_panels);
            c.take(d_last, h.brick_panels);
            c.take(d_ids, h.brick_panels);
        }
        c.take(p->d_scratch, slots * kScratchCols);
        return zero;
    };
    Carver need;
    carve(need);
    // a block the pool would not keep is the driver's: mapping it into the pool takes longer than cudaMalloc (R-MAT 2^24,
    // 3.7 GB: plan creation 130 ms longer)
    const bool pooled = need.used <= kPoolKeeps;
    if ((e = pooled ? cutespmm_internal_pool_alloc(&p->d_block, need.used, dev, s, true) : cudaMalloc(&p->d_block, need.used)) != cudaSuccess)
        return fail_cuda_status(e, "memory of the plan");
    p->block_bytes = need.used;
    if (pooled) note_live(dev, (int64_t)need.used);
    Carver c;
    c.base = static_cast<char *>(p->d_block);
    const uint64_t zero = carve(c);
    p->device_bytes = need.used;
    p->d_row_ptr = d_rp; p->d_pairs = d_pairs;
    p->d_tiles = d_tiles; p->d_chunks = d_chunks; p->d_long_rows = d_longs; p->d_chunk_owner = d_owner;
    p->d_tiles_all = d_tiles_all; p->d_chunks_all = d_chunks_all; p->d_long_rows_all = d_longs_all; p->d_chunk_owner_all = d_owner_all;
    p->d_bcols = d_bcols; p->d_brecs = d_brecs; p->d_panel_first = d_first; p->d_panel_last = d_last; p->d_panel_ids = d_ids;

    // ---- write ----
    la.tiles = bricks ? d_tiles_all : d_tiles;
    la.chunks = bricks ? d_chunks_all : d_chunks;
    la.long_rows = bricks ? d_longs_all : d_longs;
    la.owners = bricks ? d_owner_all : d_owner;
    la2.tiles = d_tiles; la2.chunks = d_chunks; la2.long_rows = d_longs; la2.owners = d_owner;
    uint32_t bad_cols = 0;
    if ((e = cudaMemsetAsync(p->d_block, 0, zero, s)) != cudaSuccess ||
        (e = launch_pack(rowPtr_dev, cols_dev, vals_dev, M, K, t.nnz, d_rp, d_pairs, &d_totals->bad_cols, sms, s)) != cudaSuccess ||
        (e = launch_lists_write(rowPtr_dev, la, s)) != cudaSuccess)
        return fail_cuda_status(e, "writing the plan");
    if (bricks) {
        // the column lists' slack behind the last slot is read, never used: any row of B will do
        if ((e = launch_lists_write(rowPtr_dev, la2, s)) != cudaSuccess ||
            (e = cudaMemsetAsync(d_bcols + h.brick_slots * kBrickCols, 0, 96 * sizeof(uint32_t), s)) != cudaSuccess ||
            (e = launch_brick_layout(P, path, ncols, ca.seg_panels, ca.seg_slots, segments, d_ids, d_first, d_last, s)) != cudaSuccess ||
            (e = launch_brick_fill(d_rp, d_pairs, M, d_ids, d_first, (uint32_t)h.brick_panels, ncols, t.brick_nnz_max, t.brick_cols_max, d_bcols, d_brecs,
                                   sms, s)) != cudaSuccess)
            return fail_cuda_status(e, "packing the bricks");
    }
    if ((e = landing.fetch(bad_cols, &d_totals->bad_cols)) != cudaSuccess)
        return fail_cuda_status(e, "packing the nonzeros");
    if (bad_cols) return fail_status(CUTESPMM_EINVAL, "column index out of range (>= K)");
    p->used_elsewhere = false;
    *plan = p;
    owner.p = nullptr;
    return CUTESPMM_OK;
}

}  // extern "C"

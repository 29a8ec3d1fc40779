// The extern "C" surface declared in include/cutespmm.h: plan life cycle, execution, sharding.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "device_plan.hpp"
#include "nvtx.hpp"
#include "plan.hpp"
#include "plan_object.hpp"

using namespace cutespmm;

namespace {
thread_local std::string g_last_error;
}
namespace cutespmm {
void set_last_error(const std::string &msg) { g_last_error = msg; }
int fail_status(int status, const std::string &msg)
{
    g_last_error = msg;
    return status;
}
int fail_cuda_status(cudaError_t e, const char *what)
{
    g_last_error = std::string(what) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? CUTESPMM_ENOMEM : CUTESPMM_ECUDA;
}
}
namespace {

int fail(int status, const std::string &msg) { return fail_status(status, msg); }
int fail_cuda(cudaError_t e, const char *what) { return fail_cuda_status(e, what); }

template <class T> cudaError_t upload(const std::vector<T> &h, void **d, uint64_t &bytes)
{
    *d = nullptr;
    if (h.empty()) return cudaSuccess;
    cudaError_t e = cudaMalloc(d, h.size() * sizeof(T));
    if (e != cudaSuccess) return e;
    bytes += h.size() * sizeof(T);
    return cudaMemcpy(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
}
}  // namespace

extern "C" {

const char *cutespmm_status_string(int status)
{
    switch (status) {
        case CUTESPMM_OK: return "success";
        case CUTESPMM_EINVAL: return "invalid argument";
        case CUTESPMM_ENOMEM: return "out of memory";
        case CUTESPMM_ECUDA: return "CUDA error";
        case CUTESPMM_EUNSUPPORTED: return "unsupported";
        case CUTESPMM_EIO: return "I/O error";
        case CUTESPMM_ETIMEOUT: return "device-side wait timed out";
        case CUTESPMM_ECOMM: return "communication library error";
        default: return "unknown status";
    }
}
const char *cutespmm_last_error(void) { return g_last_error.c_str(); }
int cutespmm_version(void) { return 100; }

static int build_common(cutespmm_plan_t **out, uint64_t M, uint64_t K, const uint64_t *rowPtr, const uint32_t *cols,
                        const float *vals, const cutespmm_options_t *opts)
{
    if (!out) return fail(CUTESPMM_EINVAL, "plan is NULL");
    *out = nullptr;
    cutespmm_plan *p = new (std::nothrow) cutespmm_plan();
    if (!p) return fail(CUTESPMM_ENOMEM, "host allocation failed");
    std::string err;
    int st;
    try {
        st = build_host_plan(p->host, M, K, rowPtr, cols, vals, opts, err);
    } catch (const std::bad_alloc &) {
        st = CUTESPMM_ENOMEM;
        err = "host allocation failed while building the plan";
    }
    if (st != CUTESPMM_OK) {
        delete p;
        return fail(st, err);
    }
    p->note_list_sizes();
    *out = p;
    return CUTESPMM_OK;
}

int cutespmm_plan_build_host(cutespmm_plan_t **plan, uint64_t M, uint64_t K, const uint64_t *rowPtr,
                             const uint32_t *cols, const float *vals, const cutespmm_options_t *opts)
{
    return build_common(plan, M, K, rowPtr, cols, vals, opts);
}

// What the row kernel needs to finish long rows inside the launch: per scratch slot the long row it belongs to (for
// both work lists), one arrival counter per long row of each list and column slab (zero between launches), and the scratch matrix.
static cudaError_t reserve_long_row_state(cutespmm_plan *p, uint64_t &by, const char **what)
{
    const HostPlan &h = p->host;
    auto owners = [](const std::vector<Chunk> &chunks, const std::vector<LongRow> &rows) {
        std::vector<uint32_t> v(chunks.size(), 0u);
        for (size_t i = 0; i < rows.size(); ++i)
            for (uint32_t k = rows[i].slot0; k < rows[i].slot1; ++k) v[k] = (uint32_t)i;
        return v;
    };
    cudaError_t e;
    *what = "chunk owners";
    if ((e = upload(owners(h.chunks, h.long_rows), &p->d_chunk_owner, by)) != cudaSuccess) return e;
    if ((e = upload(owners(h.chunks_all, h.long_rows_all), &p->d_chunk_owner_all, by)) != cudaSuccess) return e;
    const uint64_t counters = (uint64_t)(h.long_rows.size() + h.long_rows_all.size()) * kArrivalStride * sizeof(uint32_t);
    if (counters) {
        *what = "arrival counters";
        if ((e = cudaMalloc(&p->d_arrivals, counters)) != cudaSuccess || (e = cudaMemset(p->d_arrivals, 0, counters)) != cudaSuccess) return e;
        by += counters;
    }
    const uint64_t scratch = (uint64_t)std::max(h.chunks.size(), h.chunks_all.size()) * kScratchCols * sizeof(float);
    if (scratch) {
        *what = "scratch";
        if ((e = cudaMalloc(&p->d_scratch, scratch)) != cudaSuccess) return e;
        by += scratch;
    }
    return cudaSuccess;
}

// Uploads every array of a complete host-side plan to the current device and reserves scratch and status word.
static int upload_plan(cutespmm_plan *p, int dev, int sm_count)
{
    HostPlan &h = p->host;
    p->device = dev;
    p->sm_count = sm_count;
    p->on_device = true;
    uint64_t &by = p->device_bytes;
    cudaError_t e;
#define UP(vec, ptr) \
    if ((e = upload(vec, &ptr, by)) != cudaSuccess) return fail_cuda(e, "uploading " #vec);
    {   // bulk copies of a tile start/end on 16-byte boundaries: keep readable slack behind both arrays
        std::vector<uint32_t> rp(h.row_ptr);
        rp.resize(rp.size() + 8, rp.back());
        std::vector<Pair> pr(h.pairs);
        pr.resize(pr.size() + 2, Pair{0, 0});
        UP(rp, p->d_row_ptr)
        UP(pr, p->d_pairs)
    }
    UP(h.row_map, p->d_row_map)
    UP(h.tiles, p->d_tiles)
    UP(h.chunks, p->d_chunks)
    UP(h.long_rows, p->d_long_rows)
    UP(h.tiles_all, p->d_tiles_all)
    UP(h.chunks_all, p->d_chunks_all)
    UP(h.long_rows_all, p->d_long_rows_all)
    if (h.num_bricks) {
        // the producer lanes prefetch a group (4 brick slots) beyond the one in use: keep that readable
        std::vector<uint32_t> bc(h.brick_cols);
        bc.resize(bc.size() + 96, 0u);
        UP(bc, p->d_bcols)
        UP(h.brick_recs, p->d_brecs)
        UP(h.panel_first_brick, p->d_panel_first)
        UP(h.panel_last_brick, p->d_panel_last)
    }
    if (h.slab_steps) {
        std::vector<uint32_t> sc(h.slab_cols), so(h.slab_rec_off);
        sc.resize(sc.size() + 96, 0u);
        so.resize(so.size() + 16, so.back());
        UP(sc, p->d_scols)
        UP(h.slab_recs, p->d_srecs)
        UP(so, p->d_srec_off)
        UP(h.slab_first, p->d_sfirst)
        UP(h.slab_last, p->d_slast)
        UP(h.slab_ids, p->d_sids)
    }
#undef UP
    const char *what = "";
    if ((e = reserve_long_row_state(p, by, &what)) != cudaSuccess) return fail_cuda(e, what);
    if ((e = cudaMalloc(&p->d_status, 256)) != cudaSuccess || (e = cudaMemset(p->d_status, 0, 256)) != cudaSuccess)
        return fail_cuda(e, "status word");
    by += 256;
    // Clearing memory returns before it is done, and a copy from pageable memory may; both are ordered with the default stream
    // only, and the first product may be on one that does not wait for it.
    if ((e = cudaStreamSynchronize(cudaStreamLegacy)) != cudaSuccess) return fail_cuda(e, "uploading the plan");
    return CUTESPMM_OK;
}

}  // extern "C"

// for plan_io.cu: a complete host-side plan goes to the current device
int cutespmm_internal_upload_plan(cutespmm_plan *p)
{
    int dev = -1, sms = 0;
    const int st = cutespmm_internal_usable_device(&dev, &sms);
    return st != CUTESPMM_OK ? st : upload_plan(p, dev, sms);
}

extern "C" {

int cutespmm_plan_create(cutespmm_plan_t **plan, uint64_t M, uint64_t K, const uint64_t *rowPtr, const uint32_t *cols,
                         const float *vals, const cutespmm_options_t *opts)
{
    // fail before the (possibly long) host build when there is no usable device
    int dev = -1, sms = 0;
    int st = cutespmm_internal_usable_device(&dev, &sms);
    if (st != CUTESPMM_OK) return st;
    NvtxRange range("cutespmm: plan creation");
    if ((st = build_common(plan, M, K, rowPtr, cols, vals, opts)) != CUTESPMM_OK) return st;
    if ((st = upload_plan(*plan, dev, sms)) != CUTESPMM_OK) {
        delete *plan;
        *plan = nullptr;
    }
    return st;
}

int cutespmm_plan_create_u32(cutespmm_plan_t **plan, uint32_t M, uint32_t K, const uint32_t *rowPtr,
                             const uint32_t *cols, const float *vals, const cutespmm_options_t *opts)
{
    if (!rowPtr) return fail(CUTESPMM_EINVAL, "rowPtr is NULL");
    std::vector<uint64_t> rp((size_t)M + 1);
    for (size_t i = 0; i <= M; ++i) rp[i] = rowPtr[i];
    return cutespmm_plan_create(plan, M, K, rp.data(), cols, vals, opts);
}

int cutespmm_plan_destroy(cutespmm_plan_t *plan)
{
    delete plan;
    return CUTESPMM_OK;
}

int cutespmm_plan_info(const cutespmm_plan_t *p, cutespmm_plan_info_t *info)
{
    if (!p || !info) return fail(CUTESPMM_EINVAL, "null argument");
    const HostPlan &h = p->host;
    std::memset(info, 0, sizeof(*info));
    info->M = h.M; info->K = h.K; info->nnz = h.nnz;
    info->num_panels = h.num_panels();
    const int st = cutespmm_internal_fetch_views(p, nullptr, nullptr);
    if (st != CUTESPMM_OK) return st;
    info->num_blocks = h.blocked_row_ptr.empty() ? 0 : h.blocked_row_ptr.back();
    info->num_tiles = p->own.tiles;
    info->num_long_rows = p->own.long_rows;
    info->num_chunks = p->own.chunks;
    info->brick_panels = h.brick_panels;
    info->num_bricks = h.num_bricks;
    info->device_bytes = p->device_bytes;
    info->scratch_bytes_per_col = std::max(p->own.chunks, p->every.chunks) * sizeof(float);
    return CUTESPMM_OK;
}

int cutespmm_plan_dims(const cutespmm_plan_t *p, uint64_t *M, uint64_t *K, uint64_t *nnz)
{
    if (!p) return fail(CUTESPMM_EINVAL, "plan is NULL");
    if (M) *M = p->host.M;
    if (K) *K = p->host.K;
    if (nnz) *nnz = p->host.nnz;
    return CUTESPMM_OK;
}

static const char *kNoViews =
    "this plan was built on the device without the panel analysis (path rows, or a panel beyond the device sort): "
    "the panel views come with path auto / brick, or from the host builder";

static int need_views(const cutespmm_plan *p, std::vector<uint32_t> *ncols = nullptr, std::vector<uint32_t> *acols = nullptr)
{
    const int st = cutespmm_internal_fetch_views(p, ncols, acols);
    if (st != CUTESPMM_OK) return st;
    if (p->host.device_built && p->host.blocked_row_ptr.size() != p->host.num_panels() + 1) return fail(CUTESPMM_EUNSUPPORTED, kNoViews);
    return CUTESPMM_OK;
}

int cutespmm_plan_blocked_row_ptr(const cutespmm_plan_t *p, uint32_t *out)
{
    if (!p || !out) return fail(CUTESPMM_EINVAL, "null argument");
    const int st = need_views(p);
    if (st != CUTESPMM_OK) return st;
    std::memcpy(out, p->host.blocked_row_ptr.data(), p->host.blocked_row_ptr.size() * sizeof(uint32_t));
    return CUTESPMM_OK;
}
int cutespmm_plan_active_cols(const cutespmm_plan_t *p, uint32_t *out)
{
    if (!p || !out) return fail(CUTESPMM_EINVAL, "null argument");
    const HostPlan &h = p->host;
    if (!h.device_built) {
        std::memcpy(out, h.active_cols.data(), h.active_cols.size() * sizeof(uint32_t));
        return CUTESPMM_OK;
    }
    // a device-built plan does not keep the column lists: run the panel analysis and bring them back
    std::vector<uint32_t> ncols, acols;
    int st = need_views(p, &ncols, &acols);
    if (st == CUTESPMM_OK) st = cutespmm_internal_fetch_lists(p);
    if (st != CUTESPMM_OK) return st;
    const uint64_t P = h.num_panels();
    if (h.nnz == 0 || P == 0) return CUTESPMM_OK;
    for (uint64_t q = 0; q < P; ++q) {  // per panel: its columns, zero-padded to a multiple of 16 (data.cu:160,204-209)
        uint32_t *dst = out + (uint64_t)h.blocked_row_ptr[q] * kBlockCols;
        const uint32_t width = (h.blocked_row_ptr[q + 1] - h.blocked_row_ptr[q]) * kBlockCols;
        const uint32_t *src = acols.data() + h.row_ptr[q * kPanelRows];
        for (uint32_t c = 0; c < width; ++c) dst[c] = c < ncols[q] ? src[c] : 0u;
    }
    return CUTESPMM_OK;
}
int cutespmm_plan_decode_csr(const cutespmm_plan_t *p, uint64_t *rowPtr, uint32_t *cols, float *vals)
{
    if (!p || !rowPtr || (p->host.nnz && (!cols || !vals))) return fail(CUTESPMM_EINVAL, "null argument");
    if ((p->host.device_built || p->host.values_on_device) && p->on_device) {  // the current pairs live on the device, in CSR order
        const int st = cutespmm_internal_fetch_lists(p);
        if (st != CUTESPMM_OK) return st;
        const HostPlan &h = p->host;
        for (uint64_t r = 0; r <= h.M; ++r) rowPtr[r] = h.row_ptr[r];
        std::vector<Pair> pr(h.nnz);
        if (h.nnz) {
            cudaError_t e = cudaMemcpy(pr.data(), p->d_pairs, h.nnz * sizeof(Pair), cudaMemcpyDeviceToHost);
            if (e != cudaSuccess) return fail_cuda(e, "reading the packed nonzeros back");
        }
        for (uint64_t j = 0; j < h.nnz; ++j) {
            cols[j] = pr[j].col;
            std::memcpy(&vals[j], &pr[j].val_bits, 4);
        }
        return CUTESPMM_OK;
    }
    decode_host_plan(p->host, rowPtr, cols, vals);
    return CUTESPMM_OK;
}

// A small job: its long rows are cut into pieces of tens of nonzeros.
static bool short_pieces(const HostPlan &h)
{
    return item_sizes(h.nnz + kRowCost * h.M, h.nnz, h.M, 0, h.opts.split_nnz, h.opts.tile_nnz, h.adaptive_tiling).latency_bound;
}

static RowsArgs rows_args(const cutespmm_plan *p, bool all_rows, const float *B, uint64_t ldb, float *C, uint64_t ldc,
                          uint32_t N, bool b_padded, const cutespmm_item_range *rg = nullptr)
{
    const HostPlan &h = p->host;
    RowsArgs a{};
    a.row_ptr = static_cast<const uint32_t *>(p->d_row_ptr);
    a.pairs = p->d_pairs;
    a.tiles = all_rows ? p->d_tiles_all : p->d_tiles;
    a.chunks = all_rows ? p->d_chunks_all : p->d_chunks;
    a.long_rows = all_rows ? p->d_long_rows_all : p->d_long_rows;
    a.num_tiles = all_rows ? p->every.tiles : p->own.tiles;
    a.num_chunks = all_rows ? p->every.chunks : p->own.chunks;
    a.chunk_owner = static_cast<const uint32_t *>(all_rows ? p->d_chunk_owner_all : p->d_chunk_owner);
    a.arrivals = p->d_arrivals + (all_rows ? (uint64_t)p->own.long_rows * kArrivalStride : 0);
    a.dense_panels = h.num_bricks ? 1u : 0u;
    a.avg_row_nnz = (uint32_t)(h.nnz / std::max<uint64_t>(h.M, 1));
    a.short_chunks = short_pieces(h) ? 1u : 0u;
    a.B = B; a.C = C; a.scratch = p->d_scratch;
    a.ldb = ldb; a.ldc = ldc; a.ld_scratch = kScratchCols;
    a.N = N;
    a.status = p->d_status;
    a.row_map = static_cast<const uint32_t *>(p->d_row_map);
    a.uneven = a.num_chunks && h.uneven ? 1u : 0u;
    // Tiles are dealt as they are finished where there are long rows: launches of such a plan share the partial sums and must
    // not overlap anyway (where they do, their results are undefined, but the counters end at zero all the same); a plan
    // without long rows may run on several streams at once and keeps nothing between launches.
    a.counters = a.num_chunks && !rg ? p->d_status + kTileCounters : nullptr;
    a.early = h.values_on_device ? 0u : 1u;
    a.run_rows = h.run_rows;
    a.num_rows = (uint32_t)h.M;
    a.b_padded = b_padded ? 1u : 0u;
    if (rg) {  // a sub-range of the lists: 16-byte tiles and chunks (a chunk names its scratch slot and, through it, its long row)
        const uint32_t t0 = all_rows ? rg->ta0 : rg->t0, t1 = all_rows ? rg->ta1 : rg->t1;
        const uint32_t c0 = all_rows ? rg->ca0 : rg->c0, c1 = all_rows ? rg->ca1 : rg->c1;
        a.tiles = static_cast<const char *>(a.tiles) + (size_t)t0 * sizeof(Tile);
        a.chunks = static_cast<const char *>(a.chunks) + (size_t)c0 * sizeof(Chunk);
        a.num_tiles = t1 - t0;
        a.num_chunks = c1 - c0;
    }
    return a;
}
static BrickArgs brick_args(const cutespmm_plan *p, const float *B, uint64_t ldb, float *C, uint64_t ldc, uint32_t N,
                            const cutespmm_item_range *rg = nullptr)
{
    BrickArgs a{};
    a.cols = static_cast<const uint32_t *>(p->d_bcols);
    a.recs = static_cast<const uint32_t *>(p->d_brecs);
    a.panel_first = static_cast<const uint32_t *>(p->d_panel_first);
    a.panel_last = static_cast<const uint32_t *>(p->d_panel_last);
    a.num_bricks = (uint32_t)p->host.num_bricks;
    a.num_panels = (uint32_t)p->host.brick_panels;
    a.M = (uint32_t)p->host.M;
    a.K = (uint32_t)p->host.K;
    a.B = B; a.C = C;
    a.ldb = ldb; a.ldc = ldc;
    a.N = N;
    a.round_b = (p->host.opts.flags & CUTESPMM_FLAG_ROUND_B_NEAREST) ? 1u : 0u;
    a.status = p->d_status;
    a.row_map = static_cast<const uint32_t *>(p->d_row_map);
    if (rg) {  // the kernel numbers its panels from panel_first[0]: hand it the sub-list
        a.panel_first += rg->p0;
        a.panel_last += rg->p0;
        a.num_panels = rg->p1 - rg->p0;
        if (a.num_panels == 0) a.num_bricks = 0;
    }
    return a;
}

static SlabArgs slab_args(const cutespmm_plan *p, const float *B, uint64_t ldb, float *C, uint64_t ldc, uint32_t N)
{
    SlabArgs a{};
    a.cols = static_cast<const uint32_t *>(p->d_scols);
    a.recs = static_cast<const uint32_t *>(p->d_srecs);
    a.rec_off = static_cast<const uint32_t *>(p->d_srec_off);
    a.panel_first = static_cast<const uint32_t *>(p->d_sfirst);
    a.panel_last = static_cast<const uint32_t *>(p->d_slast);
    a.panel_ids = static_cast<const uint32_t *>(p->d_sids);
    a.num_panels = (uint32_t)p->host.slab_panels;
    a.M = (uint32_t)p->host.M;
    a.K = (uint32_t)p->host.K;
    a.B = B; a.C = C;
    a.ldb = ldb; a.ldc = ldc;
    a.N = N;
    a.status = p->d_status;
    return a;
}

// Whether a window of N columns at these addresses runs the brick kernel for the brick panels; if
// not, the row kernel executes every row from its all-rows work list.
// Path auto leaves products narrower than 64 columns to the row kernel even where the plan has brick panels: with a
// group of N/4 lanes per row it is the faster of the two there (stencil512 at N = 32: 0.035 against 0.041 ms,
// elasticity40: 0.045 against 0.047 ms; at N = 64 the brick kernel wins, 0.048 / 0.053 against 0.057 / 0.070 ms).
// Rows in runs of the same columns take one load per run there, and win at 64 columns too (elasticity40: 0.0405 against
// 0.0458 ms); wider, B no longer stays near the SM and the bricks win (N = 128: 0.068 against 0.063 ms).
// A plan created with path brick runs its bricks at every width the brick kernel takes.
static bool brick_wanted(const cutespmm_plan *p, uint32_t N)
{
    const HostPlan &h = p->host;
    const bool runs = h.run_rows && h.row_map.empty() && p->every.chunks == 0;
    return h.num_bricks && (N > 64 || (N == 64 && !runs) || h.opts.path == CUTESPMM_PATH_BRICK);
}
static bool use_brick(const cutespmm_plan *p, const float *B, uint64_t ldb, const float *C, uint64_t ldc, uint32_t N)
{
    return brick_wanted(p, N) && brick_supports(N, ldb, ldc, B, C);
}

int cutespmm_spmm(const cutespmm_plan_t *p, const float *B, uint64_t ldb, float *C, uint64_t ldc, uint32_t N,
                  void *stream)
{
    return cutespmm_internal_spmm_range(p, B, ldb, C, ldc, N, stream, nullptr, false);
}

}  // extern "C"

// A plan that ran on another stream than the default one is dropped with a wait for the device (its memory may be in use there).
static void note_stream(const cutespmm_plan *p, cudaStream_t s)
{
    if (s != nullptr && s != cudaStreamLegacy && !p->used_elsewhere.load(std::memory_order_relaxed)) p->used_elsewhere = true;
}

// Rows of B that are not 16-byte aligned (N not a multiple of four columns, a view) are read one or two columns per lane and load.
// Copying B once into rows of N rounded up to four first (the copy lives on the stream) costs a launch, 1.25 ps per element of the
// copy and, as C is written column by column then, 1.6 ps per element of C; with the kernels for unaligned rows as they are it
// pays in these ranges only (us without / with the copy; "graphs": rows cut into pieces, and uneven ones):
//   25 (rows in runs: 20) to 31 columns, short rows: the copy lets a warp take four rows with one load each; 6 ps per nonzero (7 per
//     row N = 31 26.0 / 21.2, stencil512 52.5 / 37.9, elasticity40 N = 22 35.5 / 31.7; 4 per row N = 27 37.9 / 46.4: not there), from 29
//     columns on 10 ps below 16 per row (100 000 x 7 N = 29 / 31 15.8 / 15.0, 16.6 / 15.2; 30 000 x 20 13.1 / 13.6: not there);
//   9 to 24 columns, 6 to 23 per row, no dense panels, 5 ps: 200 000 x 10 of 20 000 columns N = 15 / 23 25.3 / 18.7, 31.5 / 25.9, 300 000 x
//     7 of 20 000 N = 23 36.9 / 30.7 (of 300 000 N = 22 35.7 / 37.0: not there; 4 per row, of 100 000, N = 22 29.2 / 31.5); graphs
//     from 17 columns on, 4 ps, where the copy stays in L2 (R-MAT 2^18 N = 27 92.2 / 80.8, 2^20 322 / 422);
//   33 to 64 and above 256 columns (graphs: above 384), rows long enough: 0.1 ps per nonzero and column (64 per row N = 47 37.0 / 35.1,
//     N = 511 258 / 234; 100 000 x 28 of 2000 columns N = 301 260 / 239, 60 000 x 48 N = 383 396 / 338; 7 per row N = 47 32.6 / 33.9);
//   65 to 256 columns, no graph, 36 and more per row: 0.0625 ps (60 000 x 100 N = 65 / 135 / 201 / 255 160 / 141, 266 / 240, 303 / 287,
//     387 / 361, 300 000 x 40 of 20 000 columns N = 135 552 / 475; 30 000 x 60 of 300 000 columns N = 135 138 / 179: not there;
//     100 000 x 28 of 2000 N = 201 136 / 149: not there);
//   9 to 64 columns (9 to 32 where all rows are long) of jobs whose rows are even but for a few in pieces of 256: four columns per load
//     are the quickest at walking such a piece, 12 ps (400 000 x 4 and one of 1000 N = 15 35.3 / 25.1, N = 31 57.4 / 37.7, N = 47
//     62.3 / 51.7, N = 7 20.4 / 21.6; 60 000 x 32 and one of 1000 N = 15 29.3 / 25.0, N = 47 41.6 / 48.1).  Not where there are tiles
//     enough to be dealt, which hides the piece (two million x 4 and one of 3000 N = 47 206 / 231), unless all rows are long (500 000 x
//     32 and one of 3000 N = 32 195 / 174, N = 13 142 / 153);
//   65 to 256 columns of mid-sized graphs, 0.2 ps per nonzero and column against a copy that stays in L2 (R-MAT 2^15
//     with 19 per row N = 135 72.2 / 55.2, 2^16 102 / 89.0; 2^14 25.6 / 27.9 and 2^17 156 / 167: not there).
//   rows of 150 and more nonzeros at every width, in windows of columns where the copy would be too large, by 12 ps per nonzero up to
//     64 columns and 0.4 ps per nonzero and column beyond (300 per row N = 15 84.0 / 67.1, N = 301 776 / 685, 4000 x 200 per row N = 7
//     43 / 12; 120 per row N = 7 21.5 / 30.0).
// Even widths above 32 are read two columns per lane and gain nothing.  Copies above kMaxPadBytes are not made: the pool would
// give them back at every synchronisation and map them anew (1.8 GB: 4.6 -> 5.6 ms per product).  Not while the stream is being
// captured (a graph should not own memory).
constexpr uint64_t kMaxPadBytes = 512ull << 20, kNearBytes = 64ull << 20, kVeryLongRows = 150, kFewTiles = 7104;  // tiles: 8 x 148 x 6, launch_rows_t
static bool worth_padding(const cutespmm_plan *p, const cutespmm_list_sizes &list, const float *B, uint64_t ldb, const float *C, uint64_t ldc, uint32_t N)
{
    const HostPlan &h = p->host;
    const bool two = !((reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 7) && !((ldb | ldc | N) & 1);
    if ((two && N > 32) || h.K * ((uint64_t)N + 3) * sizeof(float) > kMaxPadBytes) return false;
    if (h.nnz >= kVeryLongRows * h.M) return h.nnz * (N <= 64 ? 12 : N * 2 / 5) >= 3000000 + h.K * N * 5 / 4;
    const bool graph = list.chunks && h.uneven, long_rows = h.nnz >= 24 * h.M;
    if (list.chunks && !graph && !short_pieces(h) && (list.tiles < kFewTiles || (long_rows && N > 16)) && N > 8 && N <= (long_rows ? 32u : 64u)) return h.nnz * 12 >= 3000000 + h.K * N * 5 / 4;  // picoseconds
    if (N <= 32) {
        uint32_t gain = 6;
        if (graph) {
            if (N < 17 || h.K * ((uint64_t)N + 3) * sizeof(float) > kNearBytes) return false;
            gain = 4;
        } else if (long_rows || N < (h.run_rows ? 20u : 9u)) {
            return false;
        } else if (!h.run_rows && N < 25) {
            if (h.num_bricks || h.nnz < 6 * h.M) return false;
            gain = 5;
        } else if (!h.run_rows && N > 28 && h.nnz < 16 * h.M) {
            gain = 10;
        }
        return h.nnz * gain >= 3000000 + h.K * N * 5 / 4;
    }
    if (N > 64 && N <= 256 && graph && h.K * ((uint64_t)N + 3) * sizeof(float) <= kNearBytes)
        return h.nnz * std::max(N, 100u) / 5 >= 6000000 + N * (h.K * 8 + h.M * 12) / 10;
    const bool wide = N > 64 && N <= (graph ? 384 : 256);
    if (wide && (graph || h.nnz < 36 * h.M)) return false;
    return h.nnz * N / (wide ? 16 : 10) >= 3000000 + N * (h.K * 13 + h.M * 16) / 10;
}

static bool capturing(cudaStream_t s)
{
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) == cudaSuccess) return cap != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    return true;
}

// What the next column window of a product runs, `left` columns from its end: B and C point at the window's first column.
struct ColumnWindow {
    uint32_t cols;
    bool slab, brick;  // the tensor-core panels run their kernel (otherwise the row kernel takes every row)
    bool all_rows;     // the row kernel walks its list over every row
    bool rows;         // ... and that list has entries
    bool pad;          // B is copied into padded rows first
};
// whole: not a range of the work items; may_copy() is asked only where a copy would be worth it.
template <class MayCopy>
static ColumnWindow column_window(const cutespmm_plan *p, const float *B, uint64_t ldb, const float *C, uint64_t ldc, uint32_t left, bool whole, bool b_padded,
                                  MayCopy &&may_copy)
{
    const HostPlan &h = p->host;
    ColumnWindow w{};
    w.cols = left < kScratchCols ? left : kScratchCols;
    const cutespmm_list_sizes &every = h.num_bricks || h.slab_panels ? p->every : p->own;
    // very long rows: a window is narrowed until a padded copy of it may be made
    if (h.nnz >= kVeryLongRows * h.M && ((reinterpret_cast<uintptr_t>(B) & 15) || (ldb & 3)) && h.K * ((uint64_t)w.cols + 3) * sizeof(float) > kMaxPadBytes) {
        const uint64_t fit = kMaxPadBytes / (h.K * sizeof(float)) / 128 * 128;
        if (fit && fit < w.cols && worth_padding(p, every, B, ldb, C, ldc, (uint32_t)fit) && may_copy()) w.cols = (uint32_t)fit;
    }
    w.slab = h.slab_panels && slab_supports(w.cols, ldb, ldc, B, C);
    w.brick = use_brick(p, B, ldb, C, ldc, w.cols);
    // brick panels whose shape the brick kernel does not take (N not a multiple of 32, unaligned
    // operands) are executed by the row kernel from its all-rows work list
    w.all_rows = (!w.brick && h.num_bricks) || (!w.slab && h.slab_panels);
    const cutespmm_list_sizes &list = w.all_rows ? p->every : p->own;
    w.rows = list.tiles || list.chunks;
    const bool aligned = !(reinterpret_cast<uintptr_t>(B) & 15) && !(ldb & 3) && (!(w.cols & 3) || b_padded);
    w.pad = !aligned && w.rows && whole && worth_padding(p, list, B, ldb, C, ldc, w.cols) && may_copy();
    return w;
}

// The windows of a product of N columns of contiguous operands that start on a 16-byte boundary.
template <class Fn> static void for_each_window(const cutespmm_plan *p, uint32_t N, Fn &&fn)
{
    float *at = reinterpret_cast<float *>(uintptr_t(1) << 40);  // stands for both operands, never followed
    ColumnWindow w{};
    for (uint32_t n0 = 0; n0 < N; n0 += w.cols) {
        w = column_window(p, at + n0, N, at + n0, N, N - n0, true, false, [] { return true; });
        fn(w);
    }
}

extern "C" {

int cutespmm_spmm_kernels(const cutespmm_plan_t *p, uint32_t N)
{
    if (!p || N == 0 || p->host.M == 0) return 0;
    int mask = 0;
    for_each_window(p, N, [&](const ColumnWindow &w) { mask |= (w.rows ? 1 : 0) | (w.brick ? 2 : 0) | (w.slab ? 4 : 0); });
    return mask;
}

int cutespmm_spmm_launch_count(const cutespmm_plan_t *p, uint32_t N)
{
    if (!p || N == 0 || p->host.M == 0) return 0;
    int total = 0;
    for_each_window(p, N, [&](const ColumnWindow &w) { total += (w.pad ? 1 : 0) + (w.rows ? 1 : 0) + (w.brick ? brick_launches(w.cols) : 0) + (w.slab ? 1 : 0); });
    return total;
}

}  // extern "C"

int cutespmm_internal_spmm_range(const cutespmm_plan *p, const float *B, uint64_t ldb, float *C, uint64_t ldc, uint32_t N, void *stream,
                                 const cutespmm_item_range *rg, bool b_padded)
{
    if (!p) return fail(CUTESPMM_EINVAL, "plan is NULL");
    if (!p->on_device) return fail(CUTESPMM_EUNSUPPORTED, "host-only plan: build it with cutespmm_plan_create on a CUDA device to execute it");
    if (N == 0) return CUTESPMM_OK;
    if (!C && p->host.M) return fail(CUTESPMM_EINVAL, "C is NULL");
    if (!B && p->host.nnz) return fail(CUTESPMM_EINVAL, "B is NULL");
    if (ldb < N || ldc < N) return fail(CUTESPMM_EINVAL, "leading dimension smaller than N");
    if (ldb >= (1ull << 32) || ldc >= (1ull << 32)) return fail(CUTESPMM_EUNSUPPORTED, "leading dimensions must be below 2^32 elements");
    if ((reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 3) return fail(CUTESPMM_EINVAL, "B and C must be 4-byte aligned");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (p->host.M == 0) return CUTESPMM_OK;
    int cur = -1;
    if (cudaGetDevice(&cur) != cudaSuccess || cur != p->device)
        return fail(CUTESPMM_EINVAL, "the current CUDA device (" + std::to_string(cur) + ") is not the one the plan was created on (" +
                                         std::to_string(p->device) + "): call cudaSetDevice first");
    note_stream(p, s);
    ColumnWindow w{};
    for (uint32_t n0 = 0; n0 < N; n0 += w.cols) {
        const float *Bw = B + n0;
        float *Cw = C + n0;
        w = column_window(p, Bw, ldb, Cw, ldc, N - n0, rg == nullptr, b_padded, [&] { return !capturing(s); });
        const uint32_t nw = w.cols;
        cudaError_t e;
        if (w.slab && rg) return fail(CUTESPMM_EUNSUPPORTED, "a plan with slab panels runs whole");
        if (w.slab) {
            SlabArgs sa = slab_args(p, Bw, ldb, Cw, ldc, nw);
            if ((e = launch_slab(sa, p->sm_count, s)) != cudaSuccess) return fail_cuda(e, "slab kernel launch");
        }
        if (w.brick) {
            BrickArgs ba = brick_args(p, Bw, ldb, Cw, ldc, nw, rg);
            if ((e = launch_brick(ba, p->sm_count, s)) != cudaSuccess) return fail_cuda(e, "brick kernel launch");
        }
        uint64_t ldw = ldb;
        float *copy = nullptr;
        if (w.pad) {
            ldw = (nw + 3) / 4 * 4;
            if (cutespmm_internal_pool_alloc(reinterpret_cast<void **>(&copy), p->host.K * ldw * sizeof(float), p->device, s, false) == cudaSuccess) {
                if ((e = launch_pad_rows(Bw, ldb, copy, p->host.K, nw, p->sm_count, s)) != cudaSuccess) {
                    cudaFreeAsync(copy, s);
                    return fail_cuda(e, "padding the rows of B");
                }
                Bw = copy;
            } else {  // no memory for the copy: the kernel reads B as it is, and the call waits for nothing
                cudaGetLastError();
                copy = nullptr;
                ldw = ldb;
            }
        }
        RowsArgs ra = rows_args(p, w.all_rows, Bw, ldw, Cw, ldc, nw, copy || b_padded, rg);
        e = launch_rows(ra, p->sm_count, s);
        if (copy) cudaFreeAsync(copy, s);
        if (e != cudaSuccess) return fail_cuda(e, "row kernel launch");
    }
    return CUTESPMM_OK;
}

extern "C" {

int cutespmm_sddmm(const cutespmm_plan_t *p, const float *X, uint64_t ldx, const float *Y, uint64_t ldy, uint32_t N, int scale_by_values,
                   float *out, void *stream)
{
    if (!p) return fail(CUTESPMM_EINVAL, "plan is NULL");
    if (!p->on_device) return fail(CUTESPMM_EUNSUPPORTED, "host-only plan cannot execute");
    if (!p->host.row_map.empty()) return fail(CUTESPMM_EUNSUPPORTED, "SDDMM is not available for a plan with row reordering");
    const HostPlan &h = p->host;
    if (h.nnz == 0) return CUTESPMM_OK;
    if (!out) return fail(CUTESPMM_EINVAL, "out is NULL");
    if (N && (!X || !Y)) return fail(CUTESPMM_EINVAL, "X or Y is NULL");
    if (ldx < N || ldy < N) return fail(CUTESPMM_EINVAL, "leading dimension smaller than N");
    if ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Y) | reinterpret_cast<uintptr_t>(out)) & 3)
        return fail(CUTESPMM_EINVAL, "X, Y and out must be 4-byte aligned");
    int cur = -1;
    if (cudaGetDevice(&cur) != cudaSuccess || cur != p->device)
        return fail(CUTESPMM_EINVAL, "the current CUDA device is not the one the plan was created on");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    note_stream(p, s);
    if (N == 0) {  // an empty sum
        cudaError_t e = cudaMemsetAsync(out, 0, h.nnz * sizeof(float), s);
        return e == cudaSuccess ? CUTESPMM_OK : fail_cuda(e, "cudaMemsetAsync");
    }
    const bool all = h.num_bricks || h.slab_panels;  // the work list that covers every row
    SddmmArgs a{};
    a.row_ptr = static_cast<const uint32_t *>(p->d_row_ptr);
    a.pairs = p->d_pairs;
    a.tiles = all ? p->d_tiles_all : p->d_tiles;
    a.chunks = all ? p->d_chunks_all : p->d_chunks;
    a.num_tiles = all ? p->every.tiles : p->own.tiles;
    a.num_chunks = all ? p->every.chunks : p->own.chunks;
    a.X = X; a.Y = Y; a.ldx = ldx; a.ldy = ldy; a.out = out; a.N = N;
    a.scale = scale_by_values ? 1u : 0u;
    a.short_rows = h.nnz < 4 * h.filled_rows ? 1u : 0u;
    a.early = h.values_on_device ? 0u : 1u;
    a.status = p->d_status;
    a.vec4 = !((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Y)) & 15) && !((ldx | ldy) & 3) && (ldx | ldy) < (1ull << 30) ? 1u : 0u;
    cudaError_t e = launch_sddmm(a, p->sm_count, s);
    return e == cudaSuccess ? CUTESPMM_OK : fail_cuda(e, "SDDMM kernel launch");
}

int cutespmm_plan_set_values_gathered(cutespmm_plan_t *p, const float *vals_dev, const uint32_t *order_dev, void *stream)
{
    if (!p) return fail(CUTESPMM_EINVAL, "plan is NULL");
    if (!p->on_device) return fail(CUTESPMM_EUNSUPPORTED, "host-only plan has no device arrays");
    const HostPlan &h = p->host;
    if (h.num_bricks || h.slab_panels)
        return fail(CUTESPMM_EUNSUPPORTED, "values can be replaced in a plan whose rows all run on the row kernel (path rows, or auto without dense panels)");
    if (!h.row_map.empty()) return fail(CUTESPMM_EUNSUPPORTED, "values cannot be replaced in a plan with row reordering");
    if (h.nnz == 0) return CUTESPMM_OK;
    if (!vals_dev) return fail(CUTESPMM_EINVAL, "vals is NULL");
    if ((reinterpret_cast<uintptr_t>(vals_dev) | reinterpret_cast<uintptr_t>(order_dev)) & 3) return fail(CUTESPMM_EINVAL, "vals must be 4-byte aligned");
    int cur = -1;
    if (cudaGetDevice(&cur) != cudaSuccess || cur != p->device)
        return fail(CUTESPMM_EINVAL, "the current CUDA device is not the one the plan was created on");
    note_stream(p, static_cast<cudaStream_t>(stream));
    const cudaError_t e = launch_set_values(p->d_pairs, vals_dev, order_dev, h.nnz, p->sm_count, static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return fail_cuda(e, "replacing the values");
    p->host.values_on_device = true;
    return CUTESPMM_OK;
}

int cutespmm_plan_set_values(cutespmm_plan_t *p, const float *vals_dev, void *stream)
{
    return cutespmm_plan_set_values_gathered(p, vals_dev, nullptr, stream);
}

int cutespmm_plan_csr_device(const cutespmm_plan_t *p, uint32_t *rowPtr_dev, uint32_t *cols_dev, float *vals_dev, void *stream)
{
    if (!p || !rowPtr_dev) return fail(CUTESPMM_EINVAL, "null argument");
    if (!p->on_device) return fail(CUTESPMM_EUNSUPPORTED, "host-only plan has no device arrays");
    if (!p->host.row_map.empty()) return fail(CUTESPMM_EUNSUPPORTED, "not available for a plan with row reordering");
    if (p->host.nnz && !cols_dev) return fail(CUTESPMM_EINVAL, "null argument");
    int cur = -1;
    if (cudaGetDevice(&cur) != cudaSuccess || cur != p->device)
        return fail(CUTESPMM_EINVAL, "the current CUDA device is not the one the plan was created on");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    note_stream(p, s);
    cudaError_t e = cudaMemcpyAsync(rowPtr_dev, p->d_row_ptr, (p->host.M + 1) * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) e = launch_unpack(p->d_pairs, cols_dev, vals_dev, p->host.nnz, p->sm_count, s);
    return e == cudaSuccess ? CUTESPMM_OK : fail_cuda(e, "reading the packed nonzeros");
}

int cutespmm_plan_device_status(const cutespmm_plan_t *p, uint32_t *status)
{
    if (!p || !status) return fail(CUTESPMM_EINVAL, "null argument");
    *status = 0;
    if (!p->on_device) return CUTESPMM_OK;
    cudaError_t e = cudaMemcpy(status, p->d_status, sizeof(uint32_t), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return fail_cuda(e, "reading the status word");
    // clear on read: a reported timeout does not stick to the launches that follow
    if (*status && (e = cudaMemset(p->d_status, 0, sizeof(uint32_t))) != cudaSuccess) return fail_cuda(e, "clearing the status word");
    return CUTESPMM_OK;
}

int cutespmm_partition_rows(uint64_t M, const uint64_t *rowPtr, uint32_t nparts, uint32_t align_rows, uint32_t row_cost,
                            uint64_t *bounds)
{
    std::string err;
    int st = partition_rows(M, rowPtr, nparts, align_rows, row_cost, bounds, err);
    return st == CUTESPMM_OK ? st : fail(st, err);
}

}  // extern "C"

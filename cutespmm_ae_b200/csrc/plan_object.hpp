// The plan object behind the opaque cutespmm_plan_t handle: the host-side description, the device arrays it
// owns and the streams / events / staging buffers of the host-buffer calls.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "plan.hpp"

// The 256-byte status block: word 0 the status, words kTileCounters... the row kernel's counters (RowsArgs::counters).
constexpr uint32_t kTileCounters = 16;

// A contiguous range of the plan's work items (tiles and chunks of the row kernel -- of its own list and
// of the list over every row -- and panels of the brick kernel): what one launch covers when a product is issued in
// blocks of rows.
struct cutespmm_item_range {
    uint32_t t0 = 0, t1 = 0, c0 = 0, c1 = 0;      // row kernel: tiles, chunks
    uint32_t ta0 = 0, ta1 = 0, ca0 = 0, ca1 = 0;  // the same lists over every row
    uint32_t p0 = 0, p1 = 0;                                        // brick panels (ordinals)
};
// One block of rows of the row-block host-buffer call: rows [row0, row1) of C, computed once rows [0, need) of B are
// on the device.
struct cutespmm_row_block {
    uint32_t row0 = 0, row1 = 0, need = 0;
    cutespmm_item_range items;
};

// How long the row kernel's lists are (the lists themselves may be on the device only).
struct cutespmm_list_sizes {
    uint32_t tiles = 0, chunks = 0, long_rows = 0;
};

// Gives the memory of a device-built plan back.  device_plan.cu
void cutespmm_internal_free_block(void *block, uint64_t bytes, int dev, bool used_elsewhere);

// Pinned slots that status words and sizes arrive in: handed out of pages of 256, because pinning takes milliseconds.
// Given-back slots are handed out again; the pages stay (32 KB for 256 plans that make host-buffer calls).  sharded.cu
constexpr uint32_t kStatusSlotBytes = 128;
cudaError_t cutespmm_internal_take_status_word(uint32_t **slot);
void cutespmm_internal_give_status_word(uint32_t *slot);

struct cutespmm_plan {
    cutespmm::HostPlan host;
    cutespmm_list_sizes own, every;  // of the list of the rows outside the tensor-core panels / of the list of every row
    // device-built plans: one block holds every array; the lists come to the host on demand
    void *d_block = nullptr;
    uint64_t block_bytes = 0;
    bool lists_on_host = true, views_tried = false;
    std::mutex fetch_mutex;
    mutable std::atomic<bool> used_elsewhere{false};  // ran on a stream that is not the default stream
    bool on_device = false;
    int device = -1;
    int sm_count = 0;
    uint64_t device_bytes = 0;
    // device arrays
    void *d_row_ptr = nullptr, *d_pairs = nullptr, *d_tiles = nullptr, *d_chunks = nullptr, *d_long_rows = nullptr;
    void *d_tiles_all = nullptr, *d_chunks_all = nullptr, *d_long_rows_all = nullptr;
    void *d_bcols = nullptr, *d_brecs = nullptr, *d_panel_first = nullptr, *d_panel_last = nullptr, *d_panel_ids = nullptr;
    void *d_scols = nullptr, *d_srecs = nullptr, *d_srec_off = nullptr, *d_sfirst = nullptr, *d_slast = nullptr, *d_sids = nullptr;
    void *d_row_map = nullptr;
    void *d_chunk_owner = nullptr, *d_chunk_owner_all = nullptr;  // per scratch slot: its long row
    uint32_t *d_arrivals = nullptr;  // per long row (of the own list, then of the list of every row) and column slab: chunks finished
    float *d_scratch = nullptr;
    uint32_t *d_status = nullptr;
    // staging for the host-buffer call
    float *d_B = nullptr, *d_C = nullptr;
    uint32_t *h_status = nullptr;  // pinned: where a call's status word arrives
    uint64_t staged_B = 0, staged_C = 0;
    // the host-buffer calls pipeline column windows: copy-in, exchange between ranks, product and copy-out each on a
    // stream of their own
    static constexpr int kMaxWindows = 4;
    cudaStream_t s_in = nullptr, s_x = nullptr, s_out = nullptr;
    cudaEvent_t ev_entry = nullptr, ev_done = nullptr;
    cudaEvent_t ev_in[kMaxWindows] = {}, ev_x0[kMaxWindows] = {}, ev_x1[kMaxWindows] = {}, ev_k0[kMaxWindows] = {}, ev_k1[kMaxWindows] = {};

    // the single-GPU host-buffer call in blocks of rows (banded matrices): C rows leave while later rows of B arrive
    static constexpr int kMaxRowBlocks = 16;
    std::vector<cutespmm_row_block> row_blocks;  // cut at the first such call
    bool row_blocks_tried = false;
    uint32_t row_blocks_n = 0;                   // the N they were cut for
    cudaEvent_t rb_in[kMaxRowBlocks] = {}, rb_k0[kMaxRowBlocks] = {}, rb_k1[kMaxRowBlocks] = {};

    void note_list_sizes()  // from the lists on the host
    {
        own = {(uint32_t)host.tiles.size(), (uint32_t)host.chunks.size(), (uint32_t)host.long_rows.size()};
        every = {(uint32_t)host.tiles_all.size(), (uint32_t)host.chunks_all.size(), (uint32_t)host.long_rows_all.size()};
    }

    ~cutespmm_plan()
    {
        if (!on_device) return;
        int cur = -1;
        cudaGetDevice(&cur);
        if (cur != device) cudaSetDevice(device);
        if (d_block) cutespmm_internal_free_block(d_block, block_bytes, device, used_elsewhere);
        else if (!host.device_built || lists_on_host)
            for (void *p : {d_row_ptr, d_pairs, d_tiles, d_chunks, d_long_rows, d_tiles_all, d_chunks_all, d_long_rows_all,
                            d_bcols, d_brecs, d_panel_first, d_panel_last, d_scols, d_srecs, d_srec_off, d_sfirst,
                            d_slast, d_sids, d_row_map, d_chunk_owner, d_chunk_owner_all, (void *)d_arrivals, (void *)d_scratch, (void *)d_status})
                if (p) cudaFree(p);
        for (void *p : {(void *)d_B, (void *)d_C})
            if (p) cudaFree(p);
        if (h_status) cutespmm_internal_give_status_word(h_status);
        for (cudaEvent_t ev : {ev_entry, ev_done})
            if (ev) cudaEventDestroy(ev);
        for (int w = 0; w < kMaxWindows; ++w)
            for (cudaEvent_t ev : {ev_in[w], ev_x0[w], ev_x1[w], ev_k0[w], ev_k1[w]})
                if (ev) cudaEventDestroy(ev);
        for (int i = 0; i < kMaxRowBlocks; ++i)
            for (cudaEvent_t ev : {rb_in[i], rb_k0[i], rb_k1[i]})
                if (ev) cudaEventDestroy(ev);
        for (cudaStream_t st : {s_in, s_x, s_out})
            if (st) cudaStreamDestroy(st);
        if (cur != device && cur >= 0) cudaSetDevice(cur);
    }
};


namespace cutespmm {
// shared by the translation units that implement the C ABI
int fail_status(int status, const std::string &msg);          // records the message, returns status
int fail_cuda_status(cudaError_t e, const char *what);        // same for a CUDA error
}  // namespace cutespmm

// device_plan.cu
int cutespmm_internal_usable_device(int *dev, int *sm_count);
int cutespmm_internal_fetch_lists(const cutespmm_plan *p);
int cutespmm_internal_fetch_views(const cutespmm_plan *p, std::vector<uint32_t> *ncols, std::vector<uint32_t> *acols);

// Memory of the library's pool on `dev` in the order of stream s (cudaFreeAsync gives it back).  may_wait: where there is none
// left, wait for the stream, give back what the pool keeps and try again (plan creation, which waits anyway; never a product).
cudaError_t cutespmm_internal_pool_alloc(void **p, uint64_t bytes, int dev, cudaStream_t s, bool may_wait);

// cutespmm_spmm restricted to a range of work items (nullptr: everything).  b_padded: rows of B can be read up to N rounded up
// to four columns.  capi.cu
int cutespmm_internal_spmm_range(const cutespmm_plan *p, const float *B, uint64_t ldb, float *C, uint64_t ldc, uint32_t N, void *stream,
                                 const cutespmm_item_range *range, bool b_padded);

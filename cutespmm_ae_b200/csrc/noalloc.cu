// cutespmm_spmm_csr_noalloc: the product C = A * B for callers that are not allowed to allocate.
//
// Some hosts of this library run where device memory cannot be requested at call time: inside a
// framework that has handed all of HBM to its own pool, inside a real-time loop that forbids calls
// which may synchronise the device, or in a process whose memory budget was fixed at start-up.  Such
// a caller cannot create a plan (plan creation uploads arrays and reserves the partial-sum scratch
// with cudaMalloc).  This entry point takes plain CSR arrays that already sit in device memory and
// computes the product with the row kernel's method -- a group of lanes per row, long rows cut into chunks
// whose partial sums are added in a fixed order -- keeping the partial sums in a scratch array that
// is part of the library image instead of an allocation.
//
// The scratch is the file-scope array g_scratch below (16 MiB), beside it the list of chunks and their counters
// (2 MiB).  Every GPU on which the library is loaded holds them until the process exits.  All calls on one
// device share them, and the scratch keeps whatever the previous call left there; nothing in it has to start at
// zero, because every slot a call reads was written earlier by the same call; the counters are put back to zero by the last
// block of a call.  Two calls that overlap on the same GPU (different streams, or different host threads) race on all of it
// and their results are undefined -- order them on one stream or with events -- but they stay inside their own arrays, and
// the next call that overlaps with none starts from zero counters (last_block.cuh).
//
// In host code the name g_scratch is only a stand-in, not a device address.  The address the
// kernels receive comes from cudaGetSymbolAddress, looked up once per device, with that device
// current, by the first call made on it, which also loads every kernel of this file; that first call should be made
// outside any stream capture.
//
// No counterpart in the reference project.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <string>

#include "../../include/cutespmm.h"
#include "device_plan.hpp"
#include "last_block.cuh"
#include "noalloc_rows.hpp"
#include "ptx.cuh"

namespace cutespmm {
void set_last_error(const std::string &msg);  // capi.cu
}

namespace {

namespace ptx = cutespmm::ptx;
using cutespmm::RowRange;

constexpr uint32_t kLimitSplit = CUTESPMM_NOALLOC_SPLIT_NNZ;  // the chunk length the published limit is stated for
constexpr uint64_t kScratchFloats = CUTESPMM_NOALLOC_SCRATCH_BYTES / 4;
constexpr uint32_t kListSlots = 1u << 16;                       // chunks one call can list
constexpr uint32_t kMaxSlabs = CUTESPMM_NOALLOC_MAX_N / 128;
constexpr int kWarps = 8;
constexpr uint32_t kBuf = 256;  // nonzeros a warp stages at a time
constexpr uint32_t kNoCol = 0xffffffffu;
constexpr unsigned kFull = 0xffffffffu;

static __device__ __align__(256) float g_scratch[kScratchFloats];
// {row, j0, j1, slot of the row's first chunk} of chunk i, whose partial sum is row i of the scratch
static __device__ uint4 g_list[kListSlots];
static __device__ uint32_t g_arrivals[kListSlots * kMaxSlabs];  // per first slot of a row and column slab: chunks finished
// All zero between calls: the last block of a call's main kernel puts it back, and the host where that kernel could not be
// launched behind the list.  (Clearing it on the stream in front of every call instead gives up the overlap of launches: 65 000
// nonzeros at N = 32 7.5 -> 10.3 us, R-MAT 2^16 N = 16 30.9 -> 32.9.)
struct alignas(16) State {
    uint32_t chunks, overflow;
    uint32_t mid_nnz;  // nonzeros in rows of more than MainArgs::mid that are not listed
    uint32_t balance;
    uint32_t next_row[kMaxSlabs];
};
static __device__ State g_state;

__device__ __forceinline__ RowRange load_range(const uint32_t *__restrict__ rowPtr, uint64_t r, uint32_t nnz)
{
    return cutespmm::row_range(__ldg(rowPtr + r), __ldg(rowPtr + r + 1), nnz);
}

// Lists the chunks of the rows longer than `split`.  One pass over the row pointers (4 us at 2^18 rows); which slots a row
// gets depends on the order of arrival, the order its chunks are added in does not.  A row that does not fit the list (row
// pointers that claim more nonzeros than there are) raises `overflow`: the main kernel then computes long rows whole.
// mid: not 0 where the main kernel wants to know how many nonzeros the other rows of more than `mid` hold.
__global__ void __launch_bounds__(kWarps * 32) noalloc_list_kernel(const uint32_t *__restrict__ rowPtr, uint32_t M, uint32_t nnz, uint32_t split,
                                                                   uint32_t capacity, uint32_t mid)
{
    ptx::grid_wait();
    ptx::grid_release();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint32_t in_mid = 0;
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < M; r += stride) {
        const RowRange g = load_range(rowPtr, r, nnz);
        const uint32_t len = g.j1 - g.j0;
        if (len <= split) {
            if (len > mid) in_mid += len;
            continue;
        }
        const uint32_t n = (uint32_t)(((uint64_t)len + split - 1) / split);
        const uint32_t slot0 = n <= capacity ? atomicAdd(&g_state.chunks, n) : 0u;
        if (n > capacity || slot0 > capacity - n) {
            g_state.overflow = 1;
            continue;
        }
        for (uint32_t i = 0; i < n; ++i) {
            const uint32_t j = g.j0 + i * split;
            g_list[slot0 + i] = make_uint4((uint32_t)r, j, min(g.j1 - j, split) + j, slot0);
        }
        for (uint32_t y = 0; y < kMaxSlabs; ++y) g_arrivals[slot0 * kMaxSlabs + y] = 0;
    }
    if (!mid) return;
    __shared__ uint32_t per_warp[kWarps];
    in_mid = __reduce_add_sync(kFull, in_mid);
    if (threadIdx.x % 32 == 0) per_warp[threadIdx.x / 32] = in_mid;
    __syncthreads();
    if (threadIdx.x < 32) {
        in_mid = __reduce_add_sync(kFull, threadIdx.x < kWarps ? per_warp[threadIdx.x] : 0u);
        if (threadIdx.x == 0 && in_mid) atomicAdd(&g_state.mid_nnz, in_mid);
    }
}

template <int VEC> struct Vec;
template <> struct Vec<4> { using T = float4; };
template <> struct Vec<1> { using T = float; };
__device__ __forceinline__ void zero(float4 &a) { a = make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ void zero(float &a) { a = 0.f; }
__device__ __forceinline__ void fma_to(float4 &a, float v, const float4 &b)
{
    a.x = fmaf(v, b.x, a.x); a.y = fmaf(v, b.y, a.y); a.z = fmaf(v, b.z, a.z); a.w = fmaf(v, b.w, a.w);
}
__device__ __forceinline__ void fma_to(float &a, float v, const float &b) { a = fmaf(v, b, a); }
__device__ __forceinline__ void add_to(float4 &a, const float4 &b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
__device__ __forceinline__ void add_to(float &a, const float &b) { a += b; }
__device__ __forceinline__ float4 from_lane(const float4 &a, int o)
{
    return make_float4(__shfl_xor_sync(kFull, a.x, o), __shfl_xor_sync(kFull, a.y, o), __shfl_xor_sync(kFull, a.z, o), __shfl_xor_sync(kFull, a.w, o));
}
__device__ __forceinline__ float from_lane(const float &a, int o) { return __shfl_xor_sync(kFull, a, o); }

struct MainArgs {
    const uint32_t *rowPtr, *cols;
    const float *vals, *B;
    float *C, *scratch;
    uint64_t ldb, ldc;
    uint32_t M, K, nnz, N, lds, split, capacity;  // capacity: chunks the scratch and the list hold for this call
    uint32_t claim, claim_uneven, mid;  // rows per claim, the same where rows of more than `mid` hold much of the matrix, set by launch_main
    bool whole_steps;  // whole steps of sound columns go without a check per nonzero
};

// The product.  A warp is G groups of 32/G lanes; a group spans a slab of 32/G * VEC * CH columns.  First the listed chunks
// (the groups share a chunk's nonzeros; whoever finishes a row's last chunk adds the row's slots in order and writes C),
// then the rows: a warp claims `claim` consecutive rows at a time from a counter per slab -- a fixed stride would hand the
// rows r, r + stride, ... of a power-law graph, whose long rows sit at indices with few one-bits, to the same few warps --
// and stages their nonzeros, up to kBuf at a time, in shared memory with one coalesced pass, columns checked; its groups
// then take a row each (and a long one together).  Bound by the chain of latencies of a claim (counter, row pointers, columns,
// gathers): instruction issue is 63 % busy, the L1 data pipe 45 %.  U rows of B are in flight per group, 40 warps per SM (U = 8 with 32 warps was 171 against 160 us below, then).
// R-MAT 2^18, 3.9 M nonzeros, N = 64: 815 -> 160 us (before: a warp per row and per 1024-nonzero chunk, single-column
// loads, three kernels one after the other) -> 150 (joins_batch) -> 125 (claim sizes, whole steps); R-MAT
// 2^16 N = 16 474 -> 29, uniform4096 N = 32 25.6 -> 7.5 (back to back, with overlapping launches), stencil512 N = 128 169 -> 139.
template <int VEC, int CH, int G>
__global__ void __launch_bounds__(kWarps * 32, 5) noalloc_main_kernel(MainArgs a)
{
    using V = typename Vec<VEC>::T;
    constexpr int L = 32 / G, U = (VEC == 4 ? 4 : 8) / CH;  // rows of B in flight per group
    static_assert(U >= 2 && (G == 1 || CH == 1), "groups span one vector per lane");
    constexpr bool kWhole = VEC == 1 || G <= 4;  // launch_main
    __shared__ uint2 bufs[kWarps][kBuf];
    __shared__ uint32_t starts[kWarps][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = lane / L, sub = lane % L;
    uint2 *buf = bufs[warp];
    uint32_t *start = starts[warp];
    const uint32_t col0 = blockIdx.y * (L * VEC * CH) + sub * VEC;
    bool ok[CH];
#pragma unroll
    for (int ch = 0; ch < CH; ++ch) ok[ch] = col0 + ch * L * VEC < a.N;
    const float *bl = a.B + col0;

    // nonzeros [j, j + n) to the warp's buffer; a column that is not below K counts nothing.  True: all of them are below K, and
    // whole steps are wanted.
    auto stage = [&](uint32_t j, uint32_t n) {
        bool sound = true;
        for (uint32_t t = lane; t < n; t += 32) {
            const uint32_t c = __ldg(a.cols + j + t);
            buf[t] = make_uint2(c < a.K ? c : kNoCol, __float_as_uint(__ldg(a.vals + j + t)));
            if (kWhole) sound &= c < a.K;
        }
        return kWhole && a.whole_steps && __all_sync(kFull, sound);
    };
    // acc += the staged nonzeros from, from + step, ... below end; whole steps of sound columns need no check (and a 32-bit stride)
    auto gather = [&](V(&acc)[CH], uint32_t from, uint32_t end, uint32_t step, bool sound) {
        uint32_t k = from;
        if (kWhole && sound) {
            const uint32_t ldb = (uint32_t)a.ldb;
            for (; k + (U - 1) * step < end; k += U * step) {
                uint2 pr[U];
                V x[U][CH];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    pr[u] = buf[k + u * step];
#pragma unroll
                    for (int ch = 0; ch < CH; ++ch) {
                        if (ok[ch]) x[u][ch] = __ldg(reinterpret_cast<const V *>(bl + (uint64_t)pr[u].x * ldb + ch * L * VEC));
                        else zero(x[u][ch]);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int ch = 0; ch < CH; ++ch) fma_to(acc[ch], __uint_as_float(pr[u].y), x[u][ch]);
            }
        }
        for (; k < end; k += U * step) {
            float v[U];
            V x[U][CH];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool in = k + u * step < end;
                const uint2 pr = buf[in ? k + u * step : k];
                v[u] = __uint_as_float(pr.y);
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) {
                    zero(x[u][ch]);
                    if (in && ok[ch] && pr.x != kNoCol) x[u][ch] = __ldg(reinterpret_cast<const V *>(bl + (uint64_t)pr.x * a.ldb + ch * L * VEC));
                }
                if (!in || pr.x == kNoCol) v[u] = 0.f;
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) fma_to(acc[ch], v[u], x[u][ch]);
        }
    };
    auto over_groups = [&](V(&acc)[CH]) {  // every group ends up with the sum of all groups'
#pragma unroll
        for (int o = L; o < 32; o <<= 1)
#pragma unroll
            for (int ch = 0; ch < CH; ++ch) add_to(acc[ch], from_lane(acc[ch], o));
    };
    auto store = [&](uint64_t row, const V(&acc)[CH]) {
#pragma unroll
        for (int ch = 0; ch < CH; ++ch)
            if (ok[ch]) __stcs(reinterpret_cast<V *>(a.C + row * a.ldc + col0 + ch * L * VEC), acc[ch]);
    };
    auto whole_warp = [&](V(&acc)[CH], uint32_t j0, uint32_t j1) {  // a run of nonzeros the groups share
#pragma unroll
        for (int ch = 0; ch < CH; ++ch) zero(acc[ch]);
        for (uint32_t j = j0; j < j1; j += kBuf) {
            const uint32_t n = min(kBuf, j1 - j);
            __syncwarp();
            const bool sound = stage(j, n);
            __syncwarp();
            gather(acc, grp, n, G, sound);
        }
        over_groups(acc);
    };

    ptx::grid_wait();
    ptx::grid_release();
    const bool overflow = g_state.overflow != 0, uneven = g_state.mid_nnz > a.nnz / 8;
    const uint32_t chunks = overflow ? 0u : min(g_state.chunks, a.capacity), take = chunks && uneven ? a.claim_uneven : a.claim;
    for (uint32_t c = warp * gridDim.x + blockIdx.x; c < chunks; c += gridDim.x * kWarps) {
        const uint4 ck = g_list[c];
        // a call that overlaps this one may have written the list: what it names has to lie inside this call's arrays
        if (ck.x >= a.M || ck.y > ck.z || ck.z > a.nnz || ck.w > c) continue;
        V acc[CH];
        whole_warp(acc, ck.y, ck.z);
        if (grp == 0) {
#pragma unroll
            for (int ch = 0; ch < CH; ++ch)
                if (ok[ch]) __stcg(reinterpret_cast<V *>(a.scratch + (uint64_t)c * a.lds + col0 + ch * L * VEC), acc[ch]);
        }
        __threadfence();
        __syncwarp();
        uint32_t pieces = 0;
        if (lane == 0) {
            const RowRange g = load_range(a.rowPtr, ck.x, a.nnz);
            pieces = (uint32_t)(((uint64_t)(g.j1 - g.j0) + a.split - 1) / a.split);
            if (atomicAdd(&g_arrivals[ck.w * kMaxSlabs + blockIdx.y], 1u) != pieces - 1 || pieces > a.capacity - ck.w) pieces = 0;
            __threadfence();
        }
        pieces = __shfl_sync(kFull, pieces, 0);
        if (pieces) {  // this warp finished the row's last chunk
#pragma unroll
            for (int ch = 0; ch < CH; ++ch) zero(acc[ch]);
#pragma unroll 4
            for (uint32_t k = grp; k < pieces; k += G)
#pragma unroll
                for (int ch = 0; ch < CH; ++ch)
                    if (ok[ch]) add_to(acc[ch], __ldcg(reinterpret_cast<const V *>(a.scratch + (uint64_t)(ck.w + k) * a.lds + col0 + ch * L * VEC)));
            over_groups(acc);
            if (grp == 0) store(ck.x, acc);
        }
    }

    for (;;) {
        uint32_t first = 0;
        if (lane == 0) first = atomicAdd(&g_state.next_row[blockIdx.y], take);
        first = __shfl_sync(kFull, first, 0);
        if (first >= a.M) break;
        const uint32_t cnt = min(take, a.M - first);
        RowRange g{0u, 0u};
        if ((uint32_t)lane < cnt) g = load_range(a.rowPtr, (uint64_t)first + lane, a.nnz);
        const RowRange before{__shfl_up_sync(kFull, g.j0, 1), __shfl_up_sync(kFull, g.j1, 1)};
        const bool listed = !overflow && g.j1 - g.j0 > a.split;
        for (uint32_t i0 = 0; i0 < cnt;) {
            const uint32_t j0 = __shfl_sync(kFull, g.j0, (int)i0), j1 = __shfl_sync(kFull, g.j1, (int)i0);
            if (__shfl_sync(kFull, listed, (int)i0)) {
                ++i0;
                continue;
            }
            V acc[CH];
            if (j1 - j0 > kBuf) {
                whole_warp(acc, j0, j1);
                if (grp == 0) store((uint64_t)first + i0, acc);
                ++i0;
                continue;
            }
            // the rows from i0 on whose nonzeros follow one another and fit the buffer together: what is staged up to the last
            // one's end holds all of them, so nothing below reads a position of the buffer that this batch has not written
            const bool fits = (uint32_t)lane < cnt && !listed && cutespmm::joins_batch(before, g, j0, kBuf);
            const unsigned miss = __ballot_sync(kFull, (uint32_t)lane > i0 && !fits);
            const uint32_t i1 = miss ? __ffs(miss) - 1 : 32u;
            const uint32_t end = __shfl_sync(kFull, g.j1, (int)i1 - 1);
            __syncwarp();
            const bool sound = stage(j0, end - j0);
            if ((uint32_t)lane >= i0 && (uint32_t)lane < i1) start[lane] = g.j0 - j0;
            if ((uint32_t)lane + 1 == i1) start[i1] = g.j1 - j0;
            __syncwarp();
            // a row of more than a few steps is shared by the groups, the others are a group's each
            constexpr uint32_t kShared = G == 1 ? kBuf : 4 * U;
            for (uint32_t i = i0 + grp; i < i1; i += G) {
                const uint32_t from = start[i], to = start[i + 1];
                if (G > 1 && to - from > kShared) continue;
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) zero(acc[ch]);
                gather(acc, from, to, 1, sound);
                store((uint64_t)first + i, acc);
            }
            if constexpr (G > 1) {
                __syncwarp();
                unsigned shared = __ballot_sync(kFull, (uint32_t)lane >= i0 && (uint32_t)lane < i1 && start[lane + 1] > start[lane] + kShared);
                for (; shared; shared &= shared - 1) {
                    const uint32_t i = __ffs(shared) - 1;
#pragma unroll
                    for (int ch = 0; ch < CH; ++ch) zero(acc[ch]);
                    gather(acc, start[i] + grp, start[i + 1], G, sound);
                    over_groups(acc);
                    if (grp == 0) store((uint64_t)first + i, acc);
                }
            }
            i0 = i1;
        }
    }

    __syncthreads();
    if (threadIdx.x == 0 && cutespmm::last_block_out(&g_state.balance)) {
        g_state.chunks = 0;
        g_state.overflow = 0;
        g_state.mid_nnz = 0;
        for (uint32_t y = 0; y < kMaxSlabs; ++y) g_state.next_row[y] = 0;
    }
}

template <int VEC, int CH, int G> cudaError_t launch_main(MainArgs a, int sm_count, int per_sm, cudaStream_t s)
{
    const uint32_t slabs = (a.N + 32 / G * VEC * CH - 1) / (32 / G * VEC * CH);
    const uint32_t wave = (uint32_t)(sm_count * per_sm) / slabs;  // one resident wave
    // Rows per claim: about a buffer of nonzeros; where a warp's share is two such claims, halves of it (stencil512 N = 8: 23 rows twice
    // 26.4 us, 29 and a half-empty second round 31.5).  Where an eighth of the nonzeros sits in rows of more than twice the mean
    // that are not listed, beside rows that are, a quarter of a buffer, or the warps that meet several of those end last (R-MAT 2^18
    // N = 64: 18 rows per claim 148 us, 4 rows 125; claims that shrink towards the end leave 148: the heavy ones come first).  A few
    // long rows alone are no reason, they are summed before the claims: quarters took 49.1 / 56.5 us against 28.8 / 41.7 at N = 16 /
    // 32 with 400 000 rows of 4 and one of 2000, 199 against 96 with a million rows at N = 32.  R-MAT graphs hold 17 % and more of
    // their nonzeros in such rows; counting them takes the list kernel 0.3 us, which is left out where both claims are the same.
    // (Each warp going by the rows of its last claim instead: R-MAT 2^16 N = 64 44 -> 64.)
    const uint64_t fill = std::min<uint64_t>((uint64_t)kBuf * a.M / (a.nnz + 1) + 1, 32), per_warp = (uint64_t)a.M / ((uint64_t)wave * kWarps) + 1;
    const uint64_t rounds = (per_warp + fill - 1) / fill;
    a.claim = (uint32_t)std::max<uint64_t>(rounds == 2 ? (per_warp + 1) / 2 : std::min(fill, per_warp), G);
    a.claim_uneven = (uint32_t)std::max<uint64_t>(std::min<uint64_t>(fill / 4, per_warp), G);
    // Whole steps pay in rows of several of them (32 per row N = 32 30.7 -> 28.8, R-MAT 2^18 N = 256 638 -> 355; 4 per row N = 32 39 -> 45:
    // not there), later where B does not stay in L2 (735 000 x 10 per row N = 32, 71 MB, 135 -> 151 us; stencil512 N = 64, 67 MB, 80 -> 74), and
    // not with eight groups, whose rows end at different steps (64 per row N = 8 25 -> 36); single columns per lane always gain (64
    // per row N = 47 81 -> 47, 4 per row 95 -> 75).
    const uint64_t least = (uint64_t)a.K * a.N * sizeof(float) > (64ull << 20) ? 12 : 6;
    a.whole_steps = a.ldb < (1ull << 32) && (VEC == 1 || (G <= 4 && a.nnz >= least * CH * a.M));
    a.mid = a.claim == a.claim_uneven ? 0u : (uint32_t)std::max<uint64_t>(2ull * a.nnz / a.M, 32);
    const uint64_t claim = a.claim;
    const uint64_t row_blocks = ((uint64_t)a.M + claim * kWarps - 1) / (claim * kWarps), chunk_blocks = (2ull * a.nnz / a.split + kWarps - 1) / kWarps;
    const uint64_t want = a.nnz > a.split && chunk_blocks > row_blocks ? chunk_blocks : row_blocks;
    if (a.nnz > a.split) {
        const uint64_t rows = ((uint64_t)a.M + kWarps * 32 - 1) / (kWarps * 32), cap = (uint64_t)sm_count * 8;
        const cudaError_t e = cutespmm::launch_overlapped(noalloc_list_kernel, (uint32_t)(rows < cap ? rows : cap), kWarps * 32, 0, s, a.rowPtr, a.M, a.nnz, a.split,
                                                          a.capacity, a.mid);
        if (e != cudaSuccess) return e;
    }
    return cutespmm::launch_overlapped(noalloc_main_kernel<VEC, CH, G>, dim3((uint32_t)(want < wave ? (want ? want : 1) : (wave ? wave : 1)), slabs), kWarps * 32,
                                       0, s, a);
}

// Loads the kernel's code on the current device and asks how many of its blocks an SM holds.
template <int VEC, int CH, int G> cudaError_t load_main(int *per_sm)
{
    cudaFuncAttributes attr{};
    const cudaError_t e = cudaFuncGetAttributes(&attr, noalloc_main_kernel<VEC, CH, G>);
    return e != cudaSuccess ? e : cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, noalloc_main_kernel<VEC, CH, G>, kWarps * 32, 0);
}

// The forms of the product, by whether the rows of B and C are 16-byte aligned and by width: four columns per lane (or one), and
// several rows per warp for narrow products.
struct Form {
    uint32_t widest;
    cudaError_t (*load)(int *per_sm);
    cudaError_t (*launch)(MainArgs, int sm_count, int per_sm, cudaStream_t);
};
template <int VEC, int CH, int G> constexpr Form form(uint32_t widest) { return Form{widest, load_main<VEC, CH, G>, launch_main<VEC, CH, G>}; }
constexpr int kWidths = 5;
constexpr Form kForms[2][kWidths] = {
    {form<1, 1, 4>(8), form<1, 1, 2>(16), form<1, 1, 1>(32), form<1, 2, 1>(64), form<1, 4, 1>(CUTESPMM_NOALLOC_MAX_N)},
    {form<4, 1, 8>(16), form<4, 1, 4>(32), form<4, 1, 2>(64), form<4, 1, 1>(128), form<4, 2, 1>(CUTESPMM_NOALLOC_MAX_N)}};

// What the calls on a device need to know, looked up by the first of them.  All of the kernels are loaded then, whatever the
// first call's width: later calls load nothing and ask nothing, so they run inside a capture or with no device memory left, and a
// call that is going to fail has queued nothing.
struct DeviceSetup {
    float *scratch = nullptr;
    void *state = nullptr;
    int sm_count = 0;
    int per_sm[2][kWidths] = {};
};
constexpr int kMaxDevices = 64;
DeviceSetup g_setup[kMaxDevices];
std::mutex g_setup_mutex;

cudaError_t look_up(int dev, DeviceSetup &d)
{
    cudaError_t e;
    if ((e = cudaGetSymbolAddress(reinterpret_cast<void **>(&d.scratch), g_scratch)) != cudaSuccess ||
        (e = cudaGetSymbolAddress(&d.state, g_state)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
    cudaFuncAttributes attr{};
    if ((e = cudaFuncGetAttributes(&attr, noalloc_list_kernel)) != cudaSuccess) return e;
    for (int v4 = 0; v4 < 2; ++v4)
        for (int w = 0; w < kWidths; ++w) {
            if ((e = kForms[v4][w].load(&d.per_sm[v4][w])) != cudaSuccess) return e;
            if (d.per_sm[v4][w] < 1) d.per_sm[v4][w] = 1;
        }
    return cudaSuccess;
}

int fail(int status, const std::string &msg)
{
    cutespmm::set_last_error(msg);
    return status;
}

}  // namespace

extern "C" int cutespmm_spmm_csr_noalloc(uint32_t M, uint32_t K, uint32_t nnz, const uint32_t *rowPtr_dev,
                                         const uint32_t *cols_dev, const float *vals_dev, const float *B_dev,
                                         uint64_t ldb, float *C_dev, uint64_t ldc, uint32_t N, void *stream)
{
    if (N == 0 || M == 0) return CUTESPMM_OK;
    if (!rowPtr_dev || !C_dev || (nnz && (!cols_dev || !vals_dev || !B_dev)))
        return fail(CUTESPMM_EINVAL, "cutespmm_spmm_csr_noalloc: null pointer");
    if (ldb < N || ldc < N) return fail(CUTESPMM_EINVAL, "cutespmm_spmm_csr_noalloc: leading dimension smaller than N");
    if (N > CUTESPMM_NOALLOC_MAX_N)
        return fail(CUTESPMM_EUNSUPPORTED, "cutespmm_spmm_csr_noalloc: N exceeds CUTESPMM_NOALLOC_MAX_N (" +
                                               std::to_string(CUTESPMM_NOALLOC_MAX_N) + "); call it per column window");
    const uint32_t lds = (N + 3) / 4 * 4;
    if (M > 0xfff00000u) return fail(CUTESPMM_EUNSUPPORTED, "cutespmm_spmm_csr_noalloc: the row counter leaves room for 2^32 - 2^20 rows");
    const uint64_t slots = 2ull * ((nnz + kLimitSplit - 1) / kLimitSplit) + 2;
    if (slots * lds > kScratchFloats)
        return fail(CUTESPMM_EUNSUPPORTED,
                    "cutespmm_spmm_csr_noalloc: the built-in scratch (" + std::to_string(CUTESPMM_NOALLOC_SCRATCH_BYTES >> 20) +
                        " MiB) holds (2*ceil(nnz/" + std::to_string(kLimitSplit) + ")+2) x N partial sums; this call needs " +
                        std::to_string((slots * lds * 4) >> 20) + " MiB. Use a plan (cutespmm_plan_create) or split the rows.");
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(CUTESPMM_ECUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices) return fail(CUTESPMM_EUNSUPPORTED, "cutespmm_spmm_csr_noalloc: device ordinal too large");
    DeviceSetup setup;
    {
        std::lock_guard<std::mutex> lock(g_setup_mutex);
        if (!g_setup[dev].scratch) {
            DeviceSetup found;
            if ((e = look_up(dev, found)) != cudaSuccess)
                return fail(CUTESPMM_ECUDA, std::string("cutespmm_spmm_csr_noalloc, first call on the device: ") + cudaGetErrorString(e));
            g_setup[dev] = found;
        }
        setup = g_setup[dev];
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // Chunks as short as a large job (256 nonzeros) or a latency-bound one (128) wants them, longer where the scratch or the
    // list would not hold them.
    uint64_t split = nnz > (2u << 20) ? 256 : 128;
    auto slots_of = [&](uint64_t len) { return 2ull * ((nnz + len - 1) / len) + 2; };
    while (slots_of(split) * lds > kScratchFloats || slots_of(split) > kListSlots) split *= 2;
    MainArgs a{rowPtr_dev, cols_dev, vals_dev, B_dev, C_dev, setup.scratch, ldb, ldc, M, K, nnz, N, lds, (uint32_t)split, (uint32_t)slots_of(split), 1, 1, 0, false};
    const int v4 = !((reinterpret_cast<uintptr_t>(B_dev) | reinterpret_cast<uintptr_t>(C_dev)) & 15) && !((ldb | ldc | N) & 3) ? 1 : 0;
    int w = 0;
    while (N > kForms[v4][w].widest) ++w;
    e = kForms[v4][w].launch(a, setup.sm_count, setup.per_sm[v4][w], s);
    if (e != cudaSuccess) cudaMemsetAsync(setup.state, 0, sizeof(State), s);  // a list without its product
    if (e != cudaSuccess) return fail(CUTESPMM_ECUDA, std::string("cutespmm_spmm_csr_noalloc launch: ") + cudaGetErrorString(e));
    return CUTESPMM_OK;
}

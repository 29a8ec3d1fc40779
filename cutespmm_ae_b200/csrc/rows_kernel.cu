// CUDA-core row-gather kernel: the path for rows whose 16x8 bricks are too empty to pay for a
// tensor-core contraction (power-law graphs, uniform random matrices), and the executor of long
// rows cut into chunks.
//
// In the reference every row panel goes through the brick kernel (kernel.cu:119-288), zero-filled
// bricks included; its tile splitter (inc/splitter.hpp:34-124) that would send light tiles to CUDA
// cores is never called.  Here a warp owns one row at a time: the lanes span the columns of B
// (one float4 each at N = 128, so a row of B is one coalesced 512-byte request), the row's
// (column, value) pairs are read from the block's staged tile in shared memory (tile_stage.cuh; one
// broadcast read per nonzero), and the products are accumulated in fp32 registers in storage order.
// For narrow products (N <= 64) a warp splits into G groups of lanes and owns that many rows at
// once.  In storage order, too, except that graphs of many tiles share rows of more than 16 nonzeros between the groups
// (Deal::kShared): such a row is G partial sums, of every G-th nonzero each, added in a fixed tree, as a piece of a long row is.
// Rows of B that are not 16-byte aligned are read one or two columns per lane and load, the lanes'
// columns interleaved, with as many loads in flight as the registers hold.  The eight warps of a block claim the rows of one
// scheduling tile as they go, so rows that share columns (stencils, block structure) meet in L1.  C rows are written once with streaming
// stores; nothing is read-modify-written: a long row is cut into chunks whose partial sums go to a
// scratch matrix and are added, in slot order, by whichever warp finishes the row's last chunk (one
// counter per long row), in the same launch.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "device_plan.hpp"
#include "last_block.cuh"
#include "plan.hpp"
#include "ptx.cuh"
#include "tile_stage.cuh"

namespace cutespmm {

namespace {

// Two tunings of the row kernel, chosen per launch (measured on R-MAT graphs and the 512x512 stencil at N = 128):
//   DEEP = false  4 rows of B in flight per warp, 5 blocks (40 warps) per SM: more warps hide the gather latency
//                 better than more loads per warp when rows are short and the grid is several waves of tiles long;
//   DEEP = true   8 rows in flight, 4 blocks per SM: fewer dependent steps per row, better for long rows and when
//                 the whole job is a single wave of tiles and the time is a handful of latencies.
template <bool DEEP> struct Tuning {
    // 48 registers, 40 warps per SM (the lane-group kernels spill 200 bytes at 40 registers and 48 warps: R-MAT 2^17 N = 64
    // 55.8 -> 50.8 us, 800 000 rows of 4 at N = 32 74 -> 65, R-MAT 2^20 N = 128 662 -> 647); the narrow kernels that deal
    // tiles by a counter have long rows to hide and keep 48 warps (R-MAT 2^20 N = 32, rows not shared: 266 us, 281 with 40)
    static constexpr int min_blocks(bool dyn, int G) { return DEEP ? 4 : dyn && G >= 4 ? 6 : 5; }
};
// Rows of B in flight per warp (or group): 16 (deep: 32) registers of B, eight rows at most.  Two column groups of two columns stay
// at four rows: with eight the deep form spills (4096 x 4096 with 16 per row at N = 66 3.8 -> 4.6 us).
template <int VEC, int CH, bool DEEP>
constexpr int kRowsInFlight = VEC == 2 && CH == 2 ? 4 : (DEEP ? 32 : 16) / (VEC * CH) < 8 ? (DEEP ? 32 : 16) / (VEC * CH) : 8;
constexpr uint32_t kSharedRow = 16;  // nonzeros from which the groups of a warp share a row (32: the same within 1 %, 64: 2-5 % slower)
constexpr int kWarps = kTileWarps;
constexpr unsigned kFull = 0xffffffffu;

template <int VEC> struct Vec;
template <> struct Vec<4> { using T = float4; };
template <> struct Vec<2> { using T = float2; };
template <> struct Vec<1> { using T = float; };

__device__ __forceinline__ float4 ldg_b(const float4 *p) { return __ldg(p); }
__device__ __forceinline__ float2 ldg_b(const float2 *p) { return __ldg(p); }
__device__ __forceinline__ float ldg_b(const float *p) { return __ldg(p); }

__device__ __forceinline__ void fma_vec(float4 &a, float v, const float4 &b)
{
    a.x = fmaf(v, b.x, a.x); a.y = fmaf(v, b.y, a.y); a.z = fmaf(v, b.z, a.z); a.w = fmaf(v, b.w, a.w);
}
__device__ __forceinline__ void fma_vec(float2 &a, float v, const float2 &b)
{
    a.x = fmaf(v, b.x, a.x); a.y = fmaf(v, b.y, a.y);
}
__device__ __forceinline__ void fma_vec(float &a, float v, const float &b) { a = fmaf(v, b, a); }

__device__ __forceinline__ void add_vec(float4 &a, const float4 &b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
__device__ __forceinline__ void add_vec(float2 &a, const float2 &b) { a.x += b.x; a.y += b.y; }
__device__ __forceinline__ void add_vec(float &a, const float &b) { a += b; }

__device__ __forceinline__ void zero_vec(float4 &a) { a = make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ void zero_vec(float2 &a) { a = make_float2(0.f, 0.f); }
__device__ __forceinline__ void zero_vec(float &a) { a = 0.f; }

// This lane's columns of a row of C: one vector store where C allows it, single columns up to N otherwise (C with rows that
// are not 16-byte aligned under a padded copy of B).
template <bool FULL>
__device__ __forceinline__ void store_row(float *p, const float4 &v, bool scalar, uint32_t cols)
{
    if (FULL || !scalar) {
        __stcs(reinterpret_cast<float4 *>(p), v);
    } else {
        __stcs(p, v.x);
        if (cols > 1) __stcs(p + 1, v.y);
        if (cols > 2) __stcs(p + 2, v.z);
        if (cols > 3) __stcs(p + 3, v.w);
    }
}
template <bool FULL> __device__ __forceinline__ void store_row(float *p, const float2 &v, bool, uint32_t) { __stcs(reinterpret_cast<float2 *>(p), v); }
template <bool FULL> __device__ __forceinline__ void store_row(float *p, const float &v, bool, uint32_t) { __stcs(p, v); }

// acc[ch] += sum over nonzeros [j0, j1) of val * B[col][lane's columns].  `bl` points at this lane's
// first column of row 0 of B; ok[ch] says whether the lane's ch-th column group exists (ragged N).
template <int VEC, int CH, bool FULL, bool DEEP>
__device__ __forceinline__ void accumulate(typename Vec<VEC>::T (&acc)[CH], const uint2 *__restrict__ pairs,
                                           uint32_t j0, uint32_t j1, const float *__restrict__ bl, uint64_t ldb,
                                           const bool (&ok)[CH], int lane)
{
    using V = typename Vec<VEC>::T;
    // nonzeros in flight per step.  Eight with float4 lanes in the shallow tuning spilled and gained nothing (at 40 registers); the
    // deep tuning and narrow lanes have the registers, and a deeper step shortens the chain of a latency-bound job
    constexpr int U = kRowsInFlight<VEC, CH, DEEP>;
    for (uint32_t j = j0; j < j1; j += 32) {
        const uint32_t n = min(32u, j1 - j);
        uint2 pr = make_uint2(0u, 0u);
        if ((uint32_t)lane < n) pr = __ldcs(pairs + j + lane);
        uint32_t k = 0;
        for (; k + U <= n; k += U) {
            float v[U];
            V b[U][CH];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t c = __shfl_sync(kFull, pr.x, k + u);
                v[u] = __uint_as_float(__shfl_sync(kFull, pr.y, k + u));
                const float *row = bl + (uint64_t)c * ldb;
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) {
                    if (FULL || ok[ch]) b[u][ch] = ldg_b(reinterpret_cast<const V *>(row + ch * 32 * VEC));
                    else zero_vec(b[u][ch]);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) fma_vec(acc[ch], v[u], b[u][ch]);
        }
        for (; k < n; ++k) {
            const uint32_t c = __shfl_sync(kFull, pr.x, k);
            const float v = __uint_as_float(__shfl_sync(kFull, pr.y, k));
            const float *row = bl + (uint64_t)c * ldb;
#pragma unroll
            for (int ch = 0; ch < CH; ++ch) {
                if (FULL || ok[ch]) {
                    const V b = ldg_b(reinterpret_cast<const V *>(row + ch * 32 * VEC));
                    fma_vec(acc[ch], v, b);
                }
            }
        }
    }
}

// acc[ch] += sum of val * B[col][lane's columns] over `cnt` staged (column, value) pairs, every STEP-th, UU rows of B in flight.
// TAIL: cnt may be smaller than UU; the surplus positions load the row of the last pair again (an L1 hit) and
// are left out of the sum.
template <int VEC, int CH, int L, bool FULL, int UU, bool TAIL, int STEP = 1>
__device__ __forceinline__ void row_group(typename Vec<VEC>::T (&acc)[CH], const uint2 *pairs_smem, uint32_t cnt, const float *__restrict__ bl,
                                          uint32_t ldb32, const bool (&ok)[CH])
{
    using V = typename Vec<VEC>::T;
    float v[UU];
    V b[UU][CH];
#pragma unroll
    for (int u = 0; u < UU; ++u) {
        const uint2 pr = pairs_smem[(TAIL ? min((uint32_t)u, cnt - 1) : (uint32_t)u) * STEP];  // all lanes read one address: broadcast
        v[u] = __uint_as_float(pr.y);
        const float *row = bl + (uint64_t)pr.x * ldb32;
#pragma unroll
        for (int ch = 0; ch < CH; ++ch) {
            if (FULL || ok[ch]) b[u][ch] = ldg_b(reinterpret_cast<const V *>(row + ch * L * VEC));
            else zero_vec(b[u][ch]);
        }
    }
#pragma unroll
    for (int u = 0; u < UU; ++u)
        if (!TAIL || (uint32_t)u < cnt) {
#pragma unroll
            for (int ch = 0; ch < CH; ++ch) fma_vec(acc[ch], v[u], b[u][ch]);
        }
}

// The same over any number of pairs, U rows of B in flight.  What is left of them (fewer than U) goes as one more group, so that its
// loads are in flight together instead of one after the other: positions past the end repeat the last pair and are not added.
template <int VEC, int CH, int L, bool FULL, int U, int STEP>
__device__ __forceinline__ void row_walk(typename Vec<VEC>::T (&acc)[CH], const uint2 *pairs_smem, uint32_t cnt, const float *__restrict__ bl, uint32_t ldb32,
                                         const bool (&ok)[CH])
{
    uint32_t j = 0;
    for (; j + U <= cnt; j += U) row_group<VEC, CH, L, FULL, U, false, STEP>(acc, pairs_smem + j * STEP, U, bl, ldb32, ok);
    if (const uint32_t rem = cnt - j) {
        if (rem > U / 2) row_group<VEC, CH, L, FULL, U, true, STEP>(acc, pairs_smem + j * STEP, rem, bl, ldb32, ok);
        else row_group<VEC, CH, L, FULL, U / 2, true, STEP>(acc, pairs_smem + j * STEP, rem, bl, ldb32, ok);
    }
}

// The same sum for a group of L = 32/G lanes that walks a chunk on its own (G > 1).  The group fetches L pairs with one
// coalesced load (lane i the i-th), the next L while these are in use, and hands them round with shuffles among its
// own lanes (`gmask`), so the groups of a warp may run different lengths.
template <int VEC, int CH, bool FULL, int U, int L>
__device__ __forceinline__ void accumulate_group(typename Vec<VEC>::T (&acc)[CH], const uint2 *__restrict__ pairs, uint32_t j0, uint32_t j1,
                                                 const float *__restrict__ bl, uint32_t ldb32, const bool (&ok)[CH], int sub, unsigned gmask)
{
    using V = typename Vec<VEC>::T;
    constexpr int UU = U < L ? U : L;  // rows of B in flight per step
    uint2 nxt = make_uint2(0u, 0u);
    if (j0 + sub < j1) nxt = __ldg(pairs + j0 + sub);
    for (uint32_t j = j0; j < j1; j += L) {
        const uint2 pr = nxt;
        if (j + L + sub < j1) nxt = __ldg(pairs + j + L + sub);
        const uint32_t n = min((uint32_t)L, j1 - j);
        for (uint32_t k = 0; k < n; k += UU) {
            float v[UU];
            V b[UU][CH];
#pragma unroll
            for (int u = 0; u < UU; ++u) {
                const int src = (int)min(k + u, n - 1);  // positions past the end repeat the last pair and are not added
                const uint32_t c = __shfl_sync(gmask, pr.x, src, L);
                v[u] = __uint_as_float(__shfl_sync(gmask, pr.y, src, L));
                const float *row = bl + (uint64_t)c * ldb32;
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) {
                    if (FULL || ok[ch]) b[u][ch] = ldg_b(reinterpret_cast<const V *>(row + ch * L * VEC));
                    else zero_vec(b[u][ch]);
                }
            }
#pragma unroll
            for (int u = 0; u < UU; ++u)
                if (k + u < n) {
#pragma unroll
                    for (int ch = 0; ch < CH; ++ch) fma_vec(acc[ch], v[u], b[u][ch]);
                }
        }
    }
}

// The same sum with the groups of a narrow warp sharing the nonzeros: group g takes nonzeros g, g + G, ... of every 32, so a
// chunk is 1/G as many dependent steps.  The pairs come 32 at a time with one coalesced load, the next 32 while these are
// in use.  Every group is left with its own partial sum.
template <int VEC, int CH, bool FULL, int U, int G>
__device__ __forceinline__ void accumulate_shared(typename Vec<VEC>::T (&acc)[CH], const uint2 *__restrict__ pairs, uint32_t j0, uint32_t j1,
                                                  const float *__restrict__ bl, uint32_t ldb32, const bool (&ok)[CH], int lane, int grp)
{
    using V = typename Vec<VEC>::T;
    constexpr int UU = U < 32 / G ? U : 32 / G;  // rows of B in flight per group and step
    uint2 nxt = make_uint2(0u, 0u);
    if (j0 + lane < j1) nxt = __ldcs(pairs + j0 + lane);
    for (uint32_t j = j0; j < j1; j += 32) {
        const uint2 pr = nxt;
        if (j + 32 + lane < j1) nxt = __ldcs(pairs + j + 32 + lane);
        const uint32_t n = min(32u, j1 - j);
        for (uint32_t k = 0; k < n; k += UU * G) {
            float v[UU];
            V b[UU][CH];
#pragma unroll
            for (int u = 0; u < UU; ++u) {
                const uint32_t at = k + u * G + grp;
                const int src = (int)min(at, n - 1);
                const uint32_t c = __shfl_sync(kFull, pr.x, src);
                v[u] = __uint_as_float(__shfl_sync(kFull, pr.y, src));
                if (at >= n) v[u] = 0.f;
                const float *row = bl + (uint64_t)c * ldb32;
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) {  // positions past the end load nothing and add nothing
                    if (at < n && (FULL || ok[ch])) b[u][ch] = ldg_b(reinterpret_cast<const V *>(row + ch * (32 / G) * VEC));
                    else zero_vec(b[u][ch]);
                }
            }
#pragma unroll
            for (int u = 0; u < UU; ++u)
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) fma_vec(acc[ch], v[u], b[u][ch]);
        }
    }
}

// acc = the sum over the groups of a warp, pairwise in a fixed tree (the result depends on nothing but the group size), in
// every lane.
__device__ __forceinline__ float4 from_lane(const float4 &a, int off)
{
    return make_float4(__shfl_xor_sync(kFull, a.x, off), __shfl_xor_sync(kFull, a.y, off), __shfl_xor_sync(kFull, a.z, off), __shfl_xor_sync(kFull, a.w, off));
}
__device__ __forceinline__ float2 from_lane(const float2 &a, int off) { return make_float2(__shfl_xor_sync(kFull, a.x, off), __shfl_xor_sync(kFull, a.y, off)); }
__device__ __forceinline__ float from_lane(const float &a, int off) { return __shfl_xor_sync(kFull, a, off); }
template <int L, class V, int CH> __device__ __forceinline__ void add_groups(V (&acc)[CH])
{
#pragma unroll
    for (int off = L; off < 32; off <<= 1)
#pragma unroll
        for (int ch = 0; ch < CH; ++ch) add_vec(acc[ch], from_lane(acc[ch], off));
}

// What the chunk part of the kernel needs.  The pointers bl / scratch / C already point at this lane's first column.
struct ChunkArgs {
    const uint2 *pairs;
    const uint4 *chunks;     // {row, j0, j1, slot}
    const uint4 *long_rows;  // {row of C, slot0, slot1, -}
    const uint32_t *chunk_owner;
    uint32_t *arrivals;
    const float *bl;
    float *scratch, *C;
    uint64_t ldb, ld_scratch, ldc;
    uint32_t num_chunks, N, col0;  // N: the end of the slab
    bool c_scalar;
};

// A chunk's partial sum goes to its slot of the scratch matrix, and the warp that completes a row's last outstanding chunk
// adds the slots in slot order -- so the sum does not depend on who that was -- and writes the row of C.  Nobody waits for
// anybody: whoever is not last just moves on.  A warp takes a chunk at a time (SHARE, or G = 1), or one per group.
template <int VEC, int CH, bool FULL, bool DEEP, int G, bool SHARE>
__device__ __forceinline__ void run_chunks(const ChunkArgs &a)
{
    using V = typename Vec<VEC>::T;
    constexpr int L = 32 / G, P = SHARE ? 1 : G;  // P chunks per warp
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int grp = G == 1 ? 0 : lane / L, sub = lane - grp * L;
    const bool lead = P == 1 ? lane == 0 : sub == 0;
    bool ok[CH];
#pragma unroll
    for (int ch = 0; ch < CH; ++ch) ok[ch] = FULL || (a.col0 + ch * L * VEC < a.N);
    // chunk (group) c goes to block c mod gridDim.x: spread over the SMs, and the warps of a block that got none
    // start on the block's tile at once (rows of a tile are claimed as they go, so they take over the others' share)
    const uint32_t gw = warp * gridDim.x + blockIdx.x, nw = gridDim.x * kWarps;
    for (uint64_t cw = gw; cw * P < a.num_chunks; cw += nw) {
        const uint64_t c = P == 1 ? cw : cw * P + grp;
        const bool have = P == 1 || c < a.num_chunks;
        uint4 ck = make_uint4(0u, 0u, 0u, 0u);
        if (have) ck = __ldg(a.chunks + c);
        // which long row the chunk belongs to.  The narrow kernels (small N: latency-bound jobs) ask now and use the
        // answer after the gathers; the wide ones ask when they need it and keep the registers for the gathers.
        uint32_t owner = 0;
        uint4 lr = make_uint4(0u, 0u, 0u, 0u);  // row of C, slot0, slot1
        if (G > 1 && have && lead) {
            owner = __ldg(a.chunk_owner + ck.w);
            lr = __ldg(a.long_rows + owner);
        }
        V acc[CH];
#pragma unroll
        for (int ch = 0; ch < CH; ++ch) zero_vec(acc[ch]);
        if constexpr (G == 1) {
            accumulate<VEC, CH, FULL, DEEP>(acc, a.pairs, ck.y, ck.z, a.bl, a.ldb, ok, lane);
        } else if constexpr (!SHARE) {
            accumulate_group<VEC, CH, FULL, kRowsInFlight<VEC, CH, DEEP>, L>(acc, a.pairs, ck.y, ck.z, a.bl, (uint32_t)a.ldb, ok, sub, ((1u << L) - 1u) << (grp * L));
        } else {
            accumulate_shared<VEC, CH, FULL, kRowsInFlight<VEC, CH, DEEP>, G>(acc, a.pairs, ck.y, ck.z, a.bl, (uint32_t)a.ldb, ok, lane, grp);
            add_groups<L>(acc);
        }
        if (P == 1 ? (G == 1 || grp == 0) : have) {
            float *out = a.scratch + (uint64_t)ck.w * a.ld_scratch;
#pragma unroll
            for (int ch = 0; ch < CH; ++ch)
                if (FULL || ok[ch]) __stcg(reinterpret_cast<V *>(out + ch * L * VEC), acc[ch]);
        }
        __threadfence();  // this lane's part of the slot is visible device-wide before the arrival is counted
        __syncwarp();
        uint32_t lr_row = 0, slot0 = 0, slot1 = 0;
        if (have && lead) {
            if (G == 1) {
                owner = __ldg(a.chunk_owner + ck.w);
                lr = __ldg(a.long_rows + owner);
            }
            // the counter of this row and column slab runs through 0 .. chunks - 1 and wraps: it is back at zero for the next launch,
            // also after launches of this list that overlapped (each adds as many as there are chunks, whatever its grid)
            uint32_t *cnt = a.arrivals + (uint64_t)owner * kArrivalStride + blockIdx.y;
            if (atomicInc(cnt, lr.z - lr.y - 1) == lr.z - lr.y - 1) {  // every chunk has arrived
                __threadfence();
                lr_row = lr.x; slot0 = lr.y; slot1 = lr.z;
            }
        }
        __syncwarp();
        // the whole warp adds the slots of every row it completed: group h takes slots h, h + G, ... in order
#pragma unroll
        for (int q = 0; q < P; ++q) {
            const uint32_t s0 = __shfl_sync(kFull, slot0, q * L), s1 = __shfl_sync(kFull, slot1, q * L), row = __shfl_sync(kFull, lr_row, q * L);
            if (s1 > s0) {  // the same for every lane of the warp
                constexpr int R = VEC * CH >= 8 || CH >= 4 ? 4 : 8;  // slots in flight
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) zero_vec(acc[ch]);
#pragma unroll R
                for (uint32_t k = s0 + grp; k < s1; k += G) {
#pragma unroll
                    for (int ch = 0; ch < CH; ++ch)
                        if (FULL || ok[ch]) add_vec(acc[ch], __ldcg(reinterpret_cast<const V *>(a.scratch + (uint64_t)k * a.ld_scratch + ch * L * VEC)));
                }
                if constexpr (G > 1) add_groups<L>(acc);
                if (G == 1 || grp == 0) {
                    float *crow = a.C + (uint64_t)row * a.ldc;
#pragma unroll
                    for (int ch = 0; ch < CH; ++ch)
                        if (FULL || ok[ch]) store_row<FULL>(crow + ch * L * VEC, acc[ch], a.c_scalar, a.N - a.col0 - ch * L * VEC);
                }
            }
        }
        if constexpr (G > 1) __syncwarp();
    }
}

// G = rows of A (or chunks) a warp works on at the same time: it is G groups of L = 32/G lanes, and a group spans L * VEC * CH
// columns, CH groups of L * VEC neighbouring ones.  G > 1 (narrow products): a group spans the whole row of B and owns a row of A
// of its own, so a warp keeps G times as many gathers in flight and few lanes idle.
// Which tiles a block gets: every gridDim.x-th, the next one of a counter, or that with the long rows of a tile shared by the groups.
enum Deal { kFixed, kDealt, kShared };

template <int VEC, int CH, bool FULL, bool DEEP, int G, Deal DEAL>
__global__ void __launch_bounds__(kWarps * 32, Tuning<DEEP>::min_blocks(DEAL != kFixed, G)) spmm_rows_kernel(RowsArgs a)
{
    constexpr bool DYN = DEAL != kFixed;
    static_assert(DEAL != kShared || G > 1, "rows are shared between groups");
    using V = typename Vec<VEC>::T;
    constexpr int L = 32 / G;  // lanes of a group
    const int lane = threadIdx.x & 31;
    const int grp = G == 1 ? 0 : lane / L, sub = G == 1 ? lane : lane % L;
    const uint32_t col0 = blockIdx.y * a.slab_cols + sub * VEC;          // this lane's first column
    const uint32_t end = min(a.N, (blockIdx.y + 1) * a.slab_cols);       // ... and the end of the block's slab
    bool ok[CH];
#pragma unroll
    for (int ch = 0; ch < CH; ++ch) ok[ch] = FULL || (col0 + ch * L * VEC < end);
    const float *bl = a.B + col0;
    const uint32_t ldb32 = (uint32_t)a.ldb;  // < 2^32 (checked by the caller): one 32x32->64 multiply per address
    const uint2 *pairs = reinterpret_cast<const uint2 *>(a.pairs);

    // ---- tiles: descriptor, row pointers and pairs arrive in shared memory by TMA, kTileStages deep ----
    __shared__ TileRing ring;
    const TileSource src{reinterpret_cast<const uint4 *>(a.tiles), a.row_ptr, pairs, a.num_tiles, DYN ? a.counters + 1 + blockIdx.y : nullptr};
    if (!a.early) ptx::grid_wait();
    tile_ring_start<DYN>(ring, src);
    ptx::grid_wait();
    ptx::grid_release();

    // Chunks of long rows first (the first tiles are on their way meanwhile): they are the largest single work items.
    if (a.num_chunks) {
        const ChunkArgs ca{pairs, reinterpret_cast<const uint4 *>(a.chunks), reinterpret_cast<const uint4 *>(a.long_rows), a.chunk_owner, a.arrivals, bl,
                           a.scratch + col0, a.C + col0, a.ldb, a.ld_scratch, a.ldc, a.num_chunks, end, col0, a.c_scalar != 0};
        // Narrow products: when the warps outnumber the chunks, a chunk is shared by the groups of a warp -- it is the longest
        // chain of the job (R-MAT 2^17: 4 500 chunks of 256, 64 steps of four gathers for a group at N = 64; N = 16 63.6 ->
        // 39.4 us, N = 32 70.4 -> 56.5) -- otherwise a group takes one on its own and the cost of starting and finishing a
        // chunk is paid once per G of them (R-MAT 2^20 N = 64: shared is 5 % slower).  The short pieces of a small job are shared
        // only when they leave half of the warps to the rows (R-MAT 2^12 N = 32 12.1 -> 9.2 us, 2^14 N = 64 14.3 -> 15.2).
        if (G == 1 || a.num_chunks <= gridDim.x * (a.short_chunks ? kWarps / 2 : kWarps)) run_chunks<VEC, CH, FULL, DEEP, G, true>(ca);
        else if constexpr (G > 1) run_chunks<VEC, CH, FULL, DEEP, G, false>(ca);
    }

    for (uint32_t i = 0;; ++i) {
        uint64_t t = blockIdx.x + (uint64_t)i * gridDim.x;
        if (!DYN && t >= a.num_tiles) break;
        const int s = i % kTileStages;
        if (!tile_wait(ring, i)) {
            if (lane == 0) atomicExch(a.status, 1u);  // the copy never landed: report, do not hang
            break;
        }
        if (DYN) {
            t = ring.tile[s];
            if (t == kNoTile) break;
        }
        const TileStage &st = ring.stage[s];
        const uint4 d = st.desc;
        const uint32_t rb = d.x & ~3u, jb = d.z & ~1u;
        constexpr int U = kRowsInFlight<VEC, CH, DEEP>;  // rows of B in flight per group and step
        if constexpr (DEAL == kShared) {
            // The rows of a tile are of very different lengths, and one of hundreds of nonzeros is a chain of as many steps for its group
            // while the tile has too few rows to go round.  The groups of a warp share such a row, group g takes nonzeros g, g + G,
            // ... (R-MAT 2^20 N = 8 / 16 / 32 / 64 210 / 212 / 266 / 367 us -> 187 / 176 / 250 / 357).
            auto store = [&](uint32_t r, V(&acc)[CH]) {
                const uint32_t r_out = a.row_map ? __ldg(a.row_map + r) : r;
                float *out = a.C + (uint64_t)r_out * a.ldc + col0;
#pragma unroll
                for (int ch = 0; ch < CH; ++ch)
                    if (FULL || ok[ch]) store_row<FULL>(out + ch * L * VEC, acc[ch], a.c_scalar != 0, end - col0 - ch * L * VEC);
            };
            for (;;) {
                const uint32_t first = tile_claim_rows(ring, s, (uint32_t)G, lane) + d.x;
                if (first >= d.y) break;
                const uint32_t r = first + grp;  // the group's own row
                uint32_t at = 0, cnt = 0;        // its nonzeros in the staged pair slice
                if (r < d.y) {
                    at = st.row_ptr[r - rb] - jb;
                    cnt = st.row_ptr[r - rb + 1] - jb - at;
                }
                V acc[CH];
                if (r < d.y && cnt <= kSharedRow) {
#pragma unroll
                    for (int ch = 0; ch < CH; ++ch) zero_vec(acc[ch]);
                    row_walk<VEC, CH, L, FULL, U, 1>(acc, st.pairs + at, cnt, bl, ldb32, ok);
                    store(r, acc);
                }
                for (unsigned shared = __ballot_sync(kFull, cnt > kSharedRow && sub == 0); shared; shared &= shared - 1) {
                    const int from = __ffs(shared) - 1;  // the first lane of the group whose row it is
                    const uint32_t n = __shfl_sync(kFull, cnt, from), start = __shfl_sync(kFull, at, from);
#pragma unroll
                    for (int ch = 0; ch < CH; ++ch) zero_vec(acc[ch]);
                    row_walk<VEC, CH, L, FULL, U, G>(acc, st.pairs + start + grp, (n - grp + G - 1) / G, bl, ldb32, ok);
                    __syncwarp();
                    add_groups<L>(acc);
                    if (grp == from / L) store(first + grp, acc);
                }
            }
        } else
        for (;;) {
            uint32_t r = tile_claim_rows(ring, s, (uint32_t)G, lane) + d.x;
            if (r >= d.y) break;
            r += grp;  // the group's own row
            if (G == 1 || r < d.y) {
                const uint32_t j0 = st.row_ptr[r - rb], j1 = st.row_ptr[r - rb + 1];
                V acc[CH];
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) zero_vec(acc[ch]);
                uint32_t j = j0 - jb, jend = j1 - jb;  // positions in the staged pair slice
                for (; j + U <= jend; j += U) row_group<VEC, CH, L, FULL, U, false>(acc, st.pairs + j, U, bl, ldb32, ok);
                // what is left of the row (fewer than U nonzeros) goes as one more group, so that its loads are in flight
                // together instead of one after the other: positions past the end repeat the row's last pair and are not added
                if (const uint32_t rem = jend - j) {
                    if (rem > U / 2) row_group<VEC, CH, L, FULL, U, true>(acc, st.pairs + j, rem, bl, ldb32, ok);
                    else row_group<VEC, CH, L, FULL, U / 2, true>(acc, st.pairs + j, rem, bl, ldb32, ok);
                }
                const uint32_t r_out = a.row_map ? __ldg(a.row_map + r) : r;  // a reordered plan writes the row to its place in the caller's C
                float *out = a.C + (uint64_t)r_out * a.ldc + col0;
#pragma unroll
                for (int ch = 0; ch < CH; ++ch)
                    if (FULL || ok[ch]) store_row<FULL>(out + ch * L * VEC, acc[ch], a.c_scalar != 0, end - col0 - ch * L * VEC);
            }
            if constexpr (G > 1) __syncwarp();
        }
        tile_release<DYN>(ring, src, i, t, lane);  // the last warp to leave the stage refills it
    }
    if (DYN) {
        __syncthreads();
        if (threadIdx.x == 0 && last_block_out(a.counters))
            for (uint32_t y = 0; y < kRowSlabs; ++y) a.counters[1 + y] = 0;
    }
}

template <int VEC, int CH, bool FULL, bool DEEP, int G = 1>
cudaError_t launch_rows_t(RowsArgs a, uint32_t slabs, int sm_count, cudaStream_t s)
{
    if (slabs > kRowSlabs) return cudaErrorInvalidConfiguration;  // counters per slab: arrived chunks, dealt tiles
    const uint64_t chunk_blocks = ((uint64_t)a.num_chunks + kWarps - 1) / kWarps;
    const uint64_t work = a.num_tiles > chunk_blocks ? a.num_tiles : chunk_blocks;
    auto grid = [&](int per_sm) {  // about one resident wave over all slabs
        const uint64_t want = (uint64_t)sm_count * per_sm;
        const uint64_t gx = ((work < want ? work : want) + slabs - 1) / slabs;
        return (uint32_t)(gx ? gx : 1);
    };
    // Slabs get equal shares of the grid, so they are of equal width where whole lines gain less than that: in small jobs (uniform
    // 15727 x 13804 at N = 260: 33.4 us as 256 + 4 columns, 24.5 as 132 + 128), where the last one would be less than half full
    // (64 per row N = 320 198 -> 150 us, stencil512 N = 260 277 -> 228, 7 per row N = 288 192 -> 185; 32 per row N = 448 238 as 256 +
    // 192, 268 as 224 + 224) and off the 16-byte grid, which has no whole lines to keep (64 per row N = 334 207 -> 152 us).
    constexpr uint32_t w = 32 / G * VEC * CH;
    const bool equal = VEC < 4 || (uint64_t)a.num_tiles <= (uint64_t)sm_count * 6 || a.N - (slabs - 1) * w < w / 2;
    a.slab_cols = equal ? ((a.N + slabs - 1) / slabs + 3) & ~3u : w;
    cudaError_t e = cudaSuccess;
    auto launched = [&](auto deal) {  // tiles are dealt where there are enough of them
        constexpr Deal D = decltype(deal)::value;
        int n = 0;
        if ((e = blocks_per_sm<spmm_rows_kernel<VEC, CH, FULL, DEEP, G, D>>(n, kWarps * 32)) != cudaSuccess) return true;
        if (D != kFixed && a.num_tiles < 8ull * grid(n)) return false;
        e = launch_overlapped(spmm_rows_kernel<VEC, CH, FULL, DEEP, G, D>, dim3(grid(n), slabs), kWarps * 32, 0, s, a);
        return true;
    };
    // Sharing pays in graphs of a dozen nonzeros per row and more; short rows are claimed more slowly by the kernels that can share (us
    // dealt / shared: R-MAT 2^20 with 15 per row N = 8 / 16 / 32 209 / 185, 211 / 175, 264 / 249, 2^19 with 28 199 / 183, 181 / 166, 213 /
    // 197; 2^20 with 7 136 / 145, 134 / 136, 155 / 162; two million x 4 and one of 3000 N = 16 / 32 / 64 78.5 / 84, 105 / 112, 168 / 186,
    // but N = 8 78.5 / 73.3).  Off the 16-byte grid the claims are a smaller part of the time: always shared there (two million x 4
    // N = 48 219, 232 after a padded copy and dealt; R-MAT 2^20 with 7 per row N = 16 / 48 159 / 297, before 216 / 365).
    const bool share = VEC < 4 || (a.uneven ? a.avg_row_nnz >= kWideTileRowNnz : a.N <= 8);
    if (a.counters) {
        if constexpr (G > 1) {
            if (share && launched(std::integral_constant<Deal, kShared>{})) return e;
        }
        if constexpr (G == 1 || VEC == 4) {
            if ((G == 1 || !share) && launched(std::integral_constant<Deal, kDealt>{})) return e;
        }
    }
    launched(std::integral_constant<Deal, kFixed>{});
    return e;
}

// dst (rows x quads float4, 16-byte aligned) = src (rows x N, leading dimension ld_src), padding zeroed.  Bound by memory
// (each byte once in and once out); a thread keeps its four columns and walks the rows, four in flight.
__global__ void __launch_bounds__(256) pad_rows_kernel(const float *__restrict__ src, uint64_t ld_src, float4 *__restrict__ dst, uint32_t quads, uint32_t N,
                                                       uint64_t rows)
{
    ptx::grid_wait();
    ptx::grid_release();
    const uint32_t per_block = 256 / quads, mine = threadIdx.x / quads, c = (threadIdx.x - mine * quads) * 4;
    if (mine >= per_block) return;
    const uint64_t step = (uint64_t)gridDim.x * per_block;
    for (uint64_t r = (uint64_t)blockIdx.x * per_block + mine; r < rows; r += 4 * step) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r + u * step < rows) {
                const float *p = src + (r + u * step) * ld_src + c;
                v[u].x = __ldg(p);
                if (c + 1 < N) v[u].y = __ldg(p + 1);
                if (c + 2 < N) v[u].z = __ldg(p + 2);
                if (c + 3 < N) v[u].w = __ldg(p + 3);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (r + u * step < rows) dst[(r + u * step) * quads + c / 4] = v[u];
    }
}

}  // namespace

cudaError_t launch_pad_rows(const float *src, uint64_t ld_src, float *dst, uint64_t rows, uint32_t N, int sm_count, cudaStream_t s)
{
    const uint32_t quads = (N + 3) / 4;
    if (rows == 0 || N == 0) return cudaSuccess;
    const uint64_t per_block = 256 / quads, want = (rows + 4 * per_block - 1) / (4 * per_block), cap = (uint64_t)sm_count * 8;
    return launch_overlapped(pad_rows_kernel, (uint32_t)(want < cap ? want : cap), 256, 0, s, src, ld_src, reinterpret_cast<float4 *>(dst), quads, N, rows);
}

// Picks the widest vector the pointers, leading dimensions and N allow.
constexpr uint32_t kLongRows = 24;  // nonzeros per row from which fewer, wider groups win on rows off the 16-byte grid
cudaError_t launch_rows(const RowsArgs &args, int sm_count, cudaStream_t s)
{
    RowsArgs a = args;
    if (a.num_tiles == 0 && a.num_chunks == 0) return cudaSuccess;
    const uintptr_t pb = reinterpret_cast<uintptr_t>(a.B), pc = reinterpret_cast<uintptr_t>(a.C),
                    ps = reinterpret_cast<uintptr_t>(a.scratch);
    // four columns per lane need B's rows aligned and readable to the end of the last four; C is written as it allows
    const bool v4 = !((pb | ps) & 15) && !((a.ldb | a.ld_scratch) & 3) && ((a.N & 3) == 0 || a.b_padded);
    const bool v2 = !((pb | pc | ps) & 7) && !((a.ldb | a.ldc | a.ld_scratch | a.N) & 1);
    a.c_scalar = (pc & 15) || ((a.ldc | a.N) & 3);
    const uint32_t N = a.N;
    // Rows in runs of the same columns: one load for a run (a row map writes rows elsewhere, chunks are single rows).  Jobs with
    // fewer runs than a block per SM has lane groups keep the row kernel: they need the rows to fill the machine
    // (elasticity12 at N = 64: 4.1 us, 4.3 by runs).
    const uint64_t groups = (uint64_t)sm_count * kWarps * (N <= 16 ? 8 : N <= 32 ? 4 : N <= 64 ? 2 : 1);
    if (a.run_rows && a.num_chunks == 0 && !a.row_map && a.num_rows / a.run_rows * ((N + 127) / 128) >= groups)
        return launch_block_rows(a, v4, sm_count, s);
    // deep: at most one resident wave of tiles, or long rows (R-MAT 2^24 with 300 nonzeros per row 2.19 against 2.38 ms, with 21
    // 1.88 against 1.93; with 15 R-MAT 2^20 0.652 against 0.647 and 3.4 per row 1.50 against 1.48 in favour of shallow).  Two
    // column groups per lane halve the rows in flight, and deep pays from shorter rows on: N = 256, R-MAT 2^18 (15 per row) 275
    // against 293 us, uniform with 7 per row 122.5 against 121.6; with two slabs of such groups always (7 per row, N = 260: 180
    // against 208 us, N = 384: 221 against 244).
    const bool deep = (uint64_t)a.num_tiles <= (uint64_t)sm_count * 6 || a.avg_row_nnz >= (!v4 || N <= 128 ? 20u : N <= 256 ? 10u : 0u);
    auto full = [&](uint32_t w) { return N % w == 0 && !(v4 && a.c_scalar); };
#define CUTESPMM_GO(VEC, CH)                                                                   \
    do {                                                                                       \
        const uint32_t w = 32 * VEC * CH, slabs = (N + w - 1) / w;                             \
        if (deep)                                                                              \
            return full(w) ? launch_rows_t<VEC, CH, true, true>(a, slabs, sm_count, s)          \
                                : launch_rows_t<VEC, CH, false, true>(a, slabs, sm_count, s);  \
        return full(w) ? launch_rows_t<VEC, CH, true, false>(a, slabs, sm_count, s)             \
                            : launch_rows_t<VEC, CH, false, false>(a, slabs, sm_count, s);     \
    } while (0)
    // narrow products: G rows of A per warp, a group of 32/G lanes spans the row of B
#define CUTESPMM_GROUPS(VEC, CH, G)                                                                        \
    do {                                                                                                   \
        constexpr uint32_t w = 32 / G * VEC * CH;                                                          \
        if (deep) return full(w) ? launch_rows_t<VEC, CH, true, true, G>(a, 1, sm_count, s)                \
                                 : launch_rows_t<VEC, CH, false, true, G>(a, 1, sm_count, s);              \
        return full(w) ? launch_rows_t<VEC, CH, true, false, G>(a, 1, sm_count, s)                         \
                       : launch_rows_t<VEC, CH, false, false, G>(a, 1, sm_count, s);                       \
    } while (0)
    if (v4) {
        if (N <= 16) CUTESPMM_GROUPS(4, 1, 8);
        if (N <= 32) CUTESPMM_GROUPS(4, 1, 4);
        if (N <= 64) CUTESPMM_GROUPS(4, 1, 2);
    }
    if (v4) {
        if (N > 128) CUTESPMM_GO(4, 2);
        CUTESPMM_GO(4, 1);
    }
    // Rows off the 16-byte grid: two columns per load where they lie on the 8-byte grid, one otherwise, the lanes' columns
    // interleaved.  A warp covers up to 256 columns (before: 64 of them, with two rows in flight: R-MAT 2^20 N = 203 3501 -> 1485 us,
    // N = 511 12990 -> 3984, stencil512 N = 101 133 -> 96.6) and takes several rows up to 64 (one before; N = 7 R-MAT 2^17 47.4 -> 29.0,
    // 64 per row 22.3 -> 17.4, which took a padded copy of B until then).  How many, by what was measured (us, more groups / fewer):
    //   few_rows    fewer rows than warps: one row per warp (4096 x 16 per row N = 27 3.6 / 3.0);
    //   few_groups  rows evenly long, or a small job: N = 47 64 per row 41.7 / 37.0, R-MAT 2^14 17.2 / 14.4; against them
    //               stencil512 53.9 / 82, R-MAT 2^17 67.4 / 70.6;
    //   few_long    long rows among even ones, in pieces of 256 that nothing evens out: the piece is the longest chain, and one row per
    //               warp walks it fastest (400 000 x 4 and one of 2000 N = 47 / 63 92 / 74, 133 / 86);
    //   runs_long   rows long, evenly or not: N = 7 R-MAT 2^17 35.3 / 29.0, stencil512 15.8 / 21.8; N = 27 34.0 / 27.0 with 64
    //               per row, 37.9 / 43.6 with 4;
    //   dense_panels  neighbouring rows share columns, and their gathers hit L1: N = 13 stencil512 19.5 / 26.3, 7 per row 17.3 / 14.6.
    const bool few_rows = a.num_rows < (uint32_t)sm_count * 40;
    const bool runs_long = a.uneven || a.avg_row_nnz >= kLongRows;
    const bool few_long = a.num_chunks && !a.uneven && !a.short_chunks && a.num_tiles < (uint32_t)sm_count * 48;
    const bool few_groups = few_long || a.num_rows < (uint32_t)sm_count * 160 || (!a.uneven && a.avg_row_nnz >= kLongRows);
    if (v2 && N > 32) {
        if (N > 128) CUTESPMM_GO(2, 4);
        if (N > 64) CUTESPMM_GO(2, 2);
        if (few_groups) CUTESPMM_GO(2, 1);
        CUTESPMM_GROUPS(2, 2, 2);
    }
    if (N > 128) CUTESPMM_GO(1, 8);
    if (N > 64) CUTESPMM_GO(1, 4);
    if (N > 32) {
        if (few_groups) CUTESPMM_GO(1, 2);
        CUTESPMM_GROUPS(1, 4, 2);
    }
    if (few_rows) CUTESPMM_GO(1, 1);
    if (N > 16) {
        if (runs_long) CUTESPMM_GROUPS(1, 2, 2);
        CUTESPMM_GROUPS(1, 4, 4);
    }
    if (N > 8) {
        if (a.dense_panels) CUTESPMM_GROUPS(1, 4, 8);
        CUTESPMM_GROUPS(1, 2, 4);
    }
    if (runs_long) CUTESPMM_GROUPS(1, 1, 4);
    CUTESPMM_GROUPS(1, 2, 8);
#undef CUTESPMM_GROUPS
#undef CUTESPMM_GO
}

}  // namespace cutespmm

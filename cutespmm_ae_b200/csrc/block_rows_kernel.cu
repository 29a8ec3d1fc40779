// Row kernel for matrices whose rows come in runs of R with the same columns: the degrees of freedom of a node in a
// finite-element matrix (R = 3 in 3-D elasticity).  A group of lanes takes a run at a time: a row of B is loaded once and
// multiplied into R accumulators, where the row kernel loads it R times.  The row kernel is bound by the L1 data pipe on such
// matrices (80 % busy on elasticity40 at N = 32, half of its requests hits), and that is what a shared load relieves.
// fp32, storage order: a row's result is the row kernel's, bit for bit.  Tiles and their staging are the row kernel's too
// (tile_stage.cuh); a run that a tile boundary cuts is computed in two parts.  The reference has no counterpart (its bricks
// share loads between the rows of a panel on the tensor cores, kernel.cu:119-288).
// Here the pipe is 62 % busy and instruction issue 60 % (70 % with one column per multiply-add); the rest is the gathers' latency.
// Rows of B off the 16-byte grid are read one column per load, the lanes' columns interleaved (elasticity40 N = 63 60.5 -> 51 us, N = 203
// 222 -> 165; before, after a padded copy of B or one row at a time).
// Products wider than 128 columns go in slabs of equal width, and a block walks its tile once per slab, so that nobody waits for a
// narrow last slab's blocks and the tile's rows of B are near for all of them (elasticity40 N = 300 284 -> 199 us, N = 132 130 -> 119,
// N = 511 478 -> 335; slabs side by side in the grid before, two blocks more than a wave where there were three).  Jobs of a few
// waves of tiles spread the slabs over blocks (launch_t).
// Row kernel -> here: elasticity40 N = 32 35.1 -> 25.7 us, N = 27 48.7 -> 34.2; elasticity20 N = 128 20.4 -> 12.8.
#include <cuda_runtime.h>

#include <cstdint>

#include "device_plan.hpp"
#include "plan.hpp"
#include "ptx.cuh"
#include "tile_stage.cuh"

namespace cutespmm {

namespace {

constexpr int kUnroll = 6;  // rows of B in flight per group: 4 / 6 / 8 took 27.2 / 25.7 / 28.5 us on elasticity40 at N = 32

// a += v * b.  TWO: two columns per instruction, each rounded like fmaf (the kernel is bound by instruction issue: elasticity40 N = 32
// 24.4 -> 23.4 us, N = 64 39.6 -> 38.6; with single-column loads the register pairs cost as much as they save).
template <bool TWO> __device__ __forceinline__ void fma4(float4 &a, float v, const float4 &b)
{
    if (TWO) {
        const uint64_t vv = ptx::pack2(v, v);
        const float2 lo = ptx::unpack2(ptx::fma2(vv, ptx::pack2(b.x, b.y), ptx::pack2(a.x, a.y)));
        const float2 hi = ptx::unpack2(ptx::fma2(vv, ptx::pack2(b.z, b.w), ptx::pack2(a.z, a.w)));
        a = make_float4(lo.x, lo.y, hi.x, hi.y);
    } else {
        a.x = fmaf(v, b.x, a.x); a.y = fmaf(v, b.y, a.y); a.z = fmaf(v, b.z, a.z); a.w = fmaf(v, b.w, a.w);
    }
}

// Four columns of a row of B: one load where rows are 16-byte aligned, otherwise four of columns L apart (a load instruction
// reads neighbouring columns), `cols` of the slab's columns from the lane's first on.
template <int L, bool ALIGNED> __device__ __forceinline__ float4 load4(const float *row, bool ok, uint32_t cols)
{
    if (ALIGNED) return ok ? __ldg(reinterpret_cast<const float4 *>(row)) : make_float4(0.f, 0.f, 0.f, 0.f);
    return make_float4(ok ? __ldg(row) : 0.f, L < cols ? __ldg(row + L) : 0.f, 2 * L < cols ? __ldg(row + 2 * L) : 0.f, 3 * L < cols ? __ldg(row + 3 * L) : 0.f);
}

// U columns of a run, the pairs of its rows at first[0 .. R-1] + i: U rows of B in flight.  TAIL: only the first cnt count.
template <int R, int U, bool TAIL, int L, bool ALIGNED>
__device__ __forceinline__ void run_step(float4 (&acc)[R], const uint2 *pairs, const uint32_t (&first)[R], uint32_t i, uint32_t cnt, const float *bl, uint32_t ldb,
                                         bool ok, uint32_t cols)
{
    float4 b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const uint32_t c = pairs[first[0] + i + (TAIL ? min((uint32_t)u, cnt - 1) : u)].x;
        b[u] = load4<L, ALIGNED>(bl + (uint64_t)c * ldb, ok, cols);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (!TAIL || (uint32_t)u < cnt) {
#pragma unroll
            for (int k = 0; k < R; ++k) fma4<ALIGNED>(acc[k], __uint_as_float(pairs[first[k] + i + u].y), b[u]);
        }
}

template <int R, int G, bool ALIGNED>
__global__ void __launch_bounds__(kTileWarps * 32, 4) spmm_block_rows_kernel(RowsArgs a)
{
    constexpr int L = 32 / G, U = kUnroll;
    const int lane = threadIdx.x & 31, grp = lane / L, sub = lane % L;
    const uint32_t ldb = (uint32_t)a.ldb;

    __shared__ TileRing ring;
    const TileSource src{reinterpret_cast<const uint4 *>(a.tiles), a.row_ptr, reinterpret_cast<const uint2 *>(a.pairs), a.num_tiles, nullptr};
    if (!a.early) ptx::grid_wait();
    tile_ring_start(ring, src);
    ptx::grid_wait();
    ptx::grid_release();

    for (uint32_t i = 0;; ++i) {
        const uint64_t t = blockIdx.x + (uint64_t)i * gridDim.x;
        if (t >= a.num_tiles) break;
        const int s = i % kTileStages;
        if (!tile_wait(ring, i)) {
            if (lane == 0) atomicExch(a.status, 1u);  // the copy never landed: report, do not hang
            break;
        }
        const TileStage &st = ring.stage[s];
        const uint4 d = st.desc;
        const uint32_t rb = d.x & ~3u, jb = d.z & ~1u, run0 = d.x / R, runs = (d.y + R - 1) / R - run0;
        for (;;) {
            const uint32_t claimed = tile_claim_rows(ring, s, (uint32_t)G, lane);
            // a wide product's block walks its tile once per slab of columns
            const uint32_t walk = G == 1 ? claimed / runs : 0u, slab0 = (G == 1 ? blockIdx.y + walk * gridDim.y : 0u) * a.slab_cols;
            if (G == 1 ? slab0 >= a.N : claimed >= runs) break;
            const uint32_t run = G == 1 ? claimed - walk * runs : claimed + grp;
            if (G == 1 || run < runs) {
                const uint32_t col0 = slab0 + (ALIGNED ? sub * 4 : sub);  // a lane's columns: four from here on, or every L-th
                const uint32_t end = min(a.N, slab0 + a.slab_cols);       // the slab's end
                const bool ok = col0 < end;
                const uint32_t cols = ok ? end - col0 : 0u;
                const float *bl = a.B + col0;
                const uint32_t r0 = (run0 + run) * R, lo = max(r0, d.x), hi = min(r0 + R, d.y);
                // rows of the run outside the tile stand in for a row inside it; they are not stored
                uint32_t first[R];
#pragma unroll
                for (int k = 0; k < R; ++k) first[k] = st.row_ptr[min(max(r0 + k, lo), hi - 1) - rb] - jb;
                const uint32_t len = st.row_ptr[lo + 1 - rb] - st.row_ptr[lo - rb];
                float4 acc[R];
#pragma unroll
                for (int k = 0; k < R; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                uint32_t j = 0;
                for (; j + U <= len; j += U) run_step<R, U, false, L, ALIGNED>(acc, st.pairs, first, j, U, bl, ldb, ok, cols);
                if (const uint32_t rem = len - j) {
                    if (rem > U / 2) run_step<R, U, true, L, ALIGNED>(acc, st.pairs, first, j, rem, bl, ldb, ok, cols);
                    else run_step<R, U / 2, true, L, ALIGNED>(acc, st.pairs, first, j, rem, bl, ldb, ok, cols);
                }
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    if (r0 + k < lo || r0 + k >= hi || !ok) continue;
                    float *p = a.C + (uint64_t)(r0 + k) * a.ldc + col0;
                    if (ALIGNED && !a.c_scalar) {
                        __stcs(reinterpret_cast<float4 *>(p), acc[k]);
                    } else {
                        constexpr int D = ALIGNED ? 1 : L;
                        __stcs(p, acc[k].x);
                        if (D < cols) __stcs(p + D, acc[k].y);
                        if (2 * D < cols) __stcs(p + 2 * D, acc[k].z);
                        if (3 * D < cols) __stcs(p + 3 * D, acc[k].w);
                    }
                }
            }
            if constexpr (G > 1) __syncwarp();
        }
        tile_release(ring, src, i, t, lane);
    }
}

template <int R, int G, bool ALIGNED> cudaError_t launch_t(RowsArgs a, int sm_count, cudaStream_t s)
{
    int per_sm = 0;
    const cudaError_t e = blocks_per_sm<spmm_block_rows_kernel<R, G, ALIGNED>>(per_sm, kTileWarps * 32);
    if (e != cudaSuccess) return e;
    const uint32_t slabs = (a.N + 127) / 128, wave = (uint32_t)(sm_count * per_sm), per_slab = wave / slabs ? wave / slabs : 1;
    // Up to four waves of tiles the slabs lie beside each other in the grid, in one wave of blocks: a block that walks whole tiles has
    // too few of them (walk / grid: elasticity21 N = 132 / 256 / 512 22.9 / 18.7 us, 24.3 / 19.7, 45.2 / 38.1, elasticity28 N = 300 / 512 68.5 /
    // 64.5, 95 / 85.7, but N = 132 39.4 / 41.6; from there on elasticity33 N = 260 93.9 / 101, elasticity40 176 / 201).
    const bool spread = a.num_tiles < 4 * wave;
    a.slab_cols = ((a.N + slabs - 1) / slabs + 3) & ~3u;
    return launch_overlapped(spmm_block_rows_kernel<R, G, ALIGNED>, spread ? dim3(a.num_tiles < per_slab ? a.num_tiles : per_slab, slabs) : dim3(wave), kTileWarps * 32,
                             0, s, a);
}
template <int R, bool ALIGNED> cudaError_t launch_r(const RowsArgs &a, int sm_count, cudaStream_t s)
{
    if (a.N <= 16) return launch_t<R, 8, ALIGNED>(a, sm_count, s);
    if (a.N <= 32) return launch_t<R, 4, ALIGNED>(a, sm_count, s);
    if (a.N <= 64) return launch_t<R, 2, ALIGNED>(a, sm_count, s);
    return launch_t<R, 1, ALIGNED>(a, sm_count, s);
}

}  // namespace

// Called by launch_rows for a list without chunks and a plan whose rows come in runs of a.run_rows.  aligned: B is read four
// columns per load.
cudaError_t launch_block_rows(const RowsArgs &a, bool aligned, int sm_count, cudaStream_t s)
{
    if (aligned) return a.run_rows == 3 ? launch_r<3, true>(a, sm_count, s) : launch_r<2, true>(a, sm_count, s);
    return a.run_rows == 3 ? launch_r<3, false>(a, sm_count, s) : launch_r<2, false>(a, sm_count, s);
}

}  // namespace cutespmm

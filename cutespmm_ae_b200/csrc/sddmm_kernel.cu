// SDDMM over the sparsity pattern of a plan: for every stored nonzero (r, c) of A
//
//        out[j] = (scale ? A[r][c] : 1) * sum_n X[r][n] * Y[c][n]
//
// the "edge feature" operator that accompanies SpMM in a graph layer (the reference tree carries it as
// TC-GNN's forward_ef, TC-GNN_ATC23/TCGNN_conv/TCGNN.cpp:265, and its own kernels do not have it), and
// the gradient of SpMM with respect to the values of A (dA = SDDMM(dC, B)).  Like the row kernel it is
// bound by gathering rows of Y, and it is built on the same skeleton: the block's tiles arrive in shared
// memory by TMA, warps claim work as they go, chunks of long rows are dealt over the blocks first.  A nonzero
// is a group of eight (four for N <= 16) lanes' work and a span of 16 to 128 columns, by N.  Rows of few
// nonzeros are walked flat, 32 nonzeros per claim; wide products of longer rows take a warp per row, which
// keeps its part of X in registers.  Every nonzero has its own output, so nothing is summed across work items.
// Measured (R-MAT 2^18, 3.9 M nonzeros): N = 64 212 -> 103 us (a 128-column span before, half of it idle; now bound by the L1
// data pipe, 67 % busy, and the loads behind it), N = 32 199 -> 78 us, N = 128 186 -> 167 us.
#include <cuda_runtime.h>

#include <cstdint>

#include "device_plan.hpp"
#include "plan.hpp"
#include "tile_stage.cuh"

namespace cutespmm {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr uint32_t kRowsFromNnz = 16;  // nonzeros per row from which a wide product takes a warp per row

// LANES lanes share a nonzero and cover a span of 4 * V * LANES columns of its row of Y: as V float4 each (VEC4), lane sub
// at float4 number sub, sub + LANES, ..., or as 4 V single columns where the rows are not 16-byte aligned.  FULL: N is a
// multiple of the span.
template <int LANES, int V, bool VEC4, bool FULL> struct Span {
    static constexpr int kCols = 4 * V * LANES;
    static constexpr int kGroups = 32 / LANES;                        // nonzeros per load instruction
    static constexpr int kSteps = V >= 4 ? 2 : (V == 1 ? 4 : 8 / V);  // ... and load steps in flight per warp

    static __device__ __forceinline__ void load(float4 (&v)[V], const float *row, uint32_t c0, uint32_t N, int sub)
    {
#pragma unroll
        for (int i = 0; i < V; ++i) {
            if (VEC4) {
                const uint32_t c = c0 + (uint32_t)(sub + LANES * i) * 4;
                if (FULL || c + 4 <= N) {
                    v[i] = __ldg(reinterpret_cast<const float4 *>(row + c));
                } else {
                    v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (c < N) v[i].x = __ldg(row + c);
                    if (c + 1 < N) v[i].y = __ldg(row + c + 1);
                    if (c + 2 < N) v[i].z = __ldg(row + c + 2);
                }
            } else {
                const uint32_t c = c0 + (uint32_t)(sub + LANES * 4 * i);
                v[i].x = c < N ? __ldg(row + c) : 0.f;
                v[i].y = c + LANES < N ? __ldg(row + c + LANES) : 0.f;
                v[i].z = c + 2 * LANES < N ? __ldg(row + c + 2 * LANES) : 0.f;
                v[i].w = c + 3 * LANES < N ? __ldg(row + c + 3 * LANES) : 0.f;
            }
        }
    }

    static __device__ __forceinline__ float dot(const float4 (&x)[V], const float4 (&y)[V])
    {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < V; ++i) {
            s = fmaf(x[i].x, y[i].x, s);
            s = fmaf(x[i].y, y[i].y, s);
            s = fmaf(x[i].z, y[i].z, s);
            s = fmaf(x[i].w, y[i].w, s);
        }
        return s;
    }

    // STEPS load steps, starting at nonzero k of the item: the span c0 of X[row] (in x) against the same span of the rows of
    // Y they name.  first: write; otherwise add to the earlier spans' sums.
    template <int STEPS, class PairAt>
    static __device__ __forceinline__ void step(const SddmmArgs &a, const float4 (&x)[V], PairAt pair_at, uint32_t k, uint32_t cnt, float *out, uint32_t c0,
                                                bool first, int lane)
    {
        const int sub = lane % LANES, grp = lane / LANES;
        uint2 pr[STEPS];
        float4 y[STEPS][V];
#pragma unroll
        for (int u = 0; u < STEPS; ++u) {
            const uint32_t mine = k + u * kGroups + grp;
            pr[u] = pair_at(min(mine, cnt - 1));  // positions past the end repeat the last pair (a cache hit) and are not stored
            load(y[u], a.Y + (uint64_t)pr[u].x * a.ldy, c0, a.N, sub);
        }
#pragma unroll
        for (int u = 0; u < STEPS; ++u) {
            float s = dot(x, y[u]);
#pragma unroll
            for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
            const uint32_t mine = k + u * kGroups + grp;
            if (mine < cnt && sub == 0) {
                if (a.scale) s *= __uint_as_float(pr[u].y);
                out[mine] = first ? s : out[mine] + s;
            }
        }
    }

    // Nonzeros [0, cnt) of one row (or chunk of one) whose pairs are pair_at(k) and whose outputs are out[k]: kSteps load steps
    // in flight while more than half of them are needed, then half as many.
    template <class PairAt>
    static __device__ __forceinline__ void items(const SddmmArgs &a, const float4 (&x)[V], PairAt pair_at, uint32_t cnt, float *out, uint32_t c0, bool first,
                                                 int lane)
    {
        uint32_t k = 0;
        for (; k + kGroups * (kSteps / 2) < cnt; k += kGroups * kSteps) step<kSteps>(a, x, pair_at, k, cnt, out, c0, first, lane);
        if (k < cnt) step<kSteps / 2>(a, x, pair_at, k, cnt, out, c0, first, lane);
    }

    // n <= 32 nonzeros whose pairs are pairs[k] (shared memory), the k-th in row `row` of lane k: both rows are loaded.
    // The kFlat sums a lane ends up with are added over the lanes of its group by halving: at each level a lane hands
    // half of its sums to its partner and keeps the other half, so a step costs one shuffle instead of one per level, and
    // the lanes of a group hold different nonzeros' results at the end.
    static __device__ __forceinline__ void flat(const SddmmArgs &a, uint32_t row, const uint2 *pairs, uint32_t n, float *out, uint32_t c0, bool first, int lane)
    {
        constexpr int kFlat = V == 1 ? 4 : V == 2 ? 2 : 1;  // load steps in flight: 16 to 32 registers of X and of Y
        const int sub = lane % LANES, grp = lane / LANES;
        for (uint32_t k = 0; k < n; k += kGroups * kFlat) {
            float4 x[kFlat][V], y[kFlat][V];
#pragma unroll
            for (int u = 0; u < kFlat; ++u) {
                const uint32_t from = min(k + u * kGroups + grp, n - 1);  // positions past the end repeat the last one and are not stored
                load(x[u], a.X + (uint64_t)__shfl_sync(kFull, row, (int)from) * a.ldx, c0, a.N, sub);
                load(y[u], a.Y + (uint64_t)pairs[from].x * a.ldy, c0, a.N, sub);
            }
            float s[kFlat];
#pragma unroll
            for (int u = 0; u < kFlat; ++u) s[u] = dot(x[u], y[u]);
            uint32_t mine = 0;   // which of the group's steps this lane ends up with
            bool spare = false;  // another lane holds the same
            int left = kFlat;
#pragma unroll
            for (int o = LANES / 2; o > 0; o >>= 1) {
                const bool upper = sub & o;
                if (left > 1) {
                    left /= 2;
#pragma unroll
                    for (int i = 0; i < left; ++i) {
                        const float keep = upper ? s[i + left] : s[i], give = upper ? s[i] : s[i + left];
                        s[i] = keep + __shfl_xor_sync(kFull, give, o);
                    }
                    if (upper) mine += left;
                } else {
                    s[0] += __shfl_xor_sync(kFull, s[0], o);
                    spare |= upper;
                }
            }
            mine = k + mine * kGroups + grp;
            if (mine < n && !spare) {
                float v = s[0];
                if (a.scale) v *= __uint_as_float(pairs[mine].y);
                out[mine] = first ? v : out[mine] + v;
            }
        }
    }
};

template <int LANES, int V, bool VEC4, bool FULL, bool FLAT>
__global__ void __launch_bounds__(kTileWarps * 32, FLAT || V < 3 ? 4 : 3) sddmm_kernel(SddmmArgs a)
{
    using S = Span<LANES, V, VEC4, FULL>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % LANES;
    const uint2 *pairs = reinterpret_cast<const uint2 *>(a.pairs);
    __shared__ TileRing ring;
    const TileSource src{reinterpret_cast<const uint4 *>(a.tiles), a.row_ptr, pairs, a.num_tiles, nullptr};
    if (!a.early) ptx::grid_wait();
    tile_ring_start(ring, src);
    ptx::grid_wait();
    ptx::grid_release();

    // chunks of long rows first (the tiles are on their way): chunk c goes to block c mod gridDim.x.  The pairs of a
    // chunk come 32 at a time with one coalesced load, the next 32 while these are in use.
    {
        const uint4 *chunks = reinterpret_cast<const uint4 *>(a.chunks);
        for (uint32_t c = warp * gridDim.x + blockIdx.x; c < a.num_chunks; c += gridDim.x * kTileWarps) {
            const uint4 ck = __ldg(chunks + c);  // row, j0, j1, slot
            for (uint32_t c0 = 0; c0 < a.N; c0 += S::kCols) {
                float4 x[V];
                S::load(x, a.X + (uint64_t)ck.x * a.ldx, c0, a.N, sub);
                uint2 nxt = make_uint2(0u, 0u);
                if (ck.y + lane < ck.z) nxt = __ldg(pairs + ck.y + lane);
                for (uint32_t j = ck.y; j < ck.z; j += 32) {
                    const uint2 cur = nxt;
                    if (j + 32 + lane < ck.z) nxt = __ldg(pairs + j + 32 + lane);
                    auto pair_at = [&](uint32_t k) { return make_uint2(__shfl_sync(kFull, cur.x, (int)k), __shfl_sync(kFull, cur.y, (int)k)); };
                    S::items(a, x, pair_at, min(32u, ck.z - j), a.out + j, c0, c0 == 0, lane);
                }
            }
        }
    }

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
        const uint32_t rb = d.x & ~3u, jb = d.z & ~1u;
        if constexpr (FLAT) {
            // A warp claims 32 nonzeros at a time whatever their rows: lane i looks the row of the i-th up in the staged row
            // pointers and the groups load both rows, X and Y.  Neighbouring groups mostly name the same row of X (one
            // request for all of them).
            const uint32_t cnt = d.w - d.z;
            for (;;) {
                const uint32_t k0 = tile_claim_rows(ring, s, 32u, lane);
                if (k0 >= cnt) break;
                const uint32_t n = min(32u, cnt - k0), j = d.z + min(k0 + lane, cnt - 1);
                uint32_t lo = d.x, hi = d.y;  // the row r with row_ptr[r] <= j < row_ptr[r + 1]
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (st.row_ptr[mid - rb] <= j) lo = mid; else hi = mid;
                }
                for (uint32_t c0 = 0; c0 < a.N; c0 += S::kCols) S::flat(a, lo, st.pairs + (d.z - jb + k0), n, a.out + d.z + k0, c0, c0 == 0, lane);
            }
        } else {
            for (;;) {
                const uint32_t r = tile_claim_rows(ring, s, 1u, lane) + d.x;
                if (r >= d.y) break;
                const uint32_t j0 = st.row_ptr[r - rb], j1 = st.row_ptr[r - rb + 1];
                if (j1 == j0) continue;
                const uint2 *row_pairs = st.pairs + (j0 - jb);
                auto pair_at = [&](uint32_t k) { return row_pairs[k]; };  // the lanes of a group read one address
                for (uint32_t c0 = 0; c0 < a.N; c0 += S::kCols) {
                    float4 x[V];
                    S::load(x, a.X + (uint64_t)r * a.ldx, c0, a.N, sub);
                    S::items(a, x, pair_at, j1 - j0, a.out + j0, c0, c0 == 0, lane);
                }
            }
        }
        tile_release(ring, src, i, t, lane);
    }
}

template <int LANES, int V, bool VEC4, bool FULL, bool FLAT> cudaError_t launch_sddmm_t(const SddmmArgs &a, int sm_count, cudaStream_t s)
{
    int per_sm = 0;
    const cudaError_t e = blocks_per_sm<sddmm_kernel<LANES, V, VEC4, FULL, FLAT>>(per_sm, kTileWarps * 32);
    if (e != cudaSuccess) return e;
    const uint32_t chunk_blocks = (a.num_chunks + kTileWarps - 1) / kTileWarps;
    uint32_t blocks = a.num_tiles > chunk_blocks ? a.num_tiles : chunk_blocks;
    const uint32_t cap = (uint32_t)(sm_count * per_sm);  // one resident wave
    if (blocks > cap) blocks = cap;
    return launch_overlapped(sddmm_kernel<LANES, V, VEC4, FULL, FLAT>, blocks, kTileWarps * 32, 0, s, a);
}
template <int LANES, int V> cudaError_t launch_sddmm_v(const SddmmArgs &a, int sm_count, cudaStream_t s)
{
    if (!a.vec4) return launch_sddmm_t<LANES, V, false, false, false>(a, sm_count, s);  // twice the scalar loads: X stays in registers
    const bool full = a.N % (4 * V * LANES) == 0;
    // Nonzeros flat, or a warp per row.  A row's chain of latencies (claim, pointers, X, Y, sums) is what a warp per row
    // costs, a second load per nonzero what the flat form costs.  Flat wins up to 64 columns everywhere (R-MAT 2^18 at N = 64:
    // 125 -> 111 us, stencil512 at N = 32: 86 -> 55 us); beyond, two loads of up to 512 bytes per nonzero fill the L1 data
    // pipe, and rows of 16 and more nonzeros repay their latencies (N = 128, flat against rows: 8 per row 47 / 53 us, 16 per
    // row 78 / 71 us, elasticity40 186 / 152 us, R-MAT 2^18 170 / 190 us).
    if constexpr (V >= 3)
        if (a.avg_row_nnz >= kRowsFromNnz)
            return full ? launch_sddmm_t<LANES, V, true, true, false>(a, sm_count, s) : launch_sddmm_t<LANES, V, true, false, false>(a, sm_count, s);
    return full ? launch_sddmm_t<LANES, V, true, true, true>(a, sm_count, s) : launch_sddmm_t<LANES, V, true, false, true>(a, sm_count, s);
}

}  // namespace

cudaError_t launch_sddmm(const SddmmArgs &a, int sm_count, cudaStream_t s)
{
    if (a.num_tiles == 0 && a.num_chunks == 0) return cudaSuccess;
    // the span that covers N with the fewest idle lanes: a narrow product keeps more nonzeros in flight
    if (a.N <= 16) return launch_sddmm_v<4, 1>(a, sm_count, s);
    if (a.N <= 32) return launch_sddmm_v<8, 1>(a, sm_count, s);
    if (a.N <= 64) return launch_sddmm_v<8, 2>(a, sm_count, s);
    if (a.N <= 96) return launch_sddmm_v<8, 3>(a, sm_count, s);
    return launch_sddmm_v<8, 4>(a, sm_count, s);
}

}  // namespace cutespmm

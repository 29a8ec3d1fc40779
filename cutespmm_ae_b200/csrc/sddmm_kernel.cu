// SDDMM over the sparsity pattern of a plan: for every stored nonzero (r, c) of A
//
//        out[j] = (scale ? A[r][c] : 1) * sum_n X[r][n] * Y[c][n]
//
// the "edge feature" operator that accompanies SpMM in a graph layer (the reference tree carries it as
// TC-GNN's forward_ef, TC-GNN_ATC23/TCGNN_conv/TCGNN.cpp:265, and its own kernels do not have it), and
// the gradient of SpMM with respect to the values of A (dA = SDDMM(dC, B)).  Like the row kernel it is
// bound by gathering rows of Y, and it is built on the same skeleton: the block's tiles arrive in shared
// memory by TMA, warps claim work as they go, chunks of long rows are dealt over the blocks first.  A nonzero is a group of
// eight (four for N <= 16) lanes' work and a span of 16 to 128 columns, by N.  A warp claims 32 nonzeros whatever their rows
// and its groups walk a run of them each, a row of X in registers for as long as it lasts.  Every nonzero has its own output,
// so nothing is summed across work items.
// Bound by the latency of the gathers (32 warps per SM, 16 to 32 registers of Y in flight each) and the instructions around
// them; gathers alone would take 50 us on R-MAT 2^18 (3.9 M nonzeros) at N = 64 (20 TB/s out of L2, measured).  Before, every
// nonzero loaded its row of X again and wide products of longer rows took a warp per row: R-MAT 2^18 at N = 16 / 32 / 64 / 128
// 48.0 / 74.8 / 106 / 168 -> 43.0 / 57.1 / 83.3 / 139 us, elasticity40 N = 64 106 -> 80.7, 60 000 x 32 per row N = 64 50.6 ->
// 39.5.  Tried: the next batch's rows of Y in flight beside this one's (83 -> 86 us), the next claim looked up meanwhile (86), 40
// and 48 warps per SM with fewer rows in flight (90, 96), the tiles' rows of X prefetched into L2 (87).
#include <cuda_runtime.h>

#include <cstdint>

#include "device_plan.hpp"
#include "plan.hpp"
#include "tile_stage.cuh"

namespace cutespmm {

namespace {

constexpr unsigned kFull = 0xffffffffu;

// LANES lanes share a nonzero and cover a span of 4 * V * LANES columns of its row of Y: as V float4 each (VEC4), lane sub
// at float4 number sub, sub + LANES, ..., or as 4 V single columns where the rows are not 16-byte aligned.  FULL: N is a
// multiple of the span.
// EACH: a row of X is loaded beside every row of Y, for matrices whose rows are so short that a group hardly meets one twice.
template <int LANES, int V, bool VEC4, bool FULL, bool EACH> struct Span {
    static constexpr int kCols = 4 * V * LANES;
    static constexpr int kGroups = 32 / LANES;                        // nonzeros per load instruction
    static constexpr unsigned kGroupStarts = LANES == 8 ? 0x01010101u : 0x11111111u;  // the first lane of every group
    static constexpr int kSteps = 2;                                  // ... and load steps in flight per warp that walks a row

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

    // Row r of X or Y.  Four columns per lane: `ld` is below 2^30 (SddmmArgs::vec4), so the stride in bytes is 32 bits wide and an
    // address is one 32 x 32 + 64-bit multiply-add.
    static __device__ __forceinline__ const float *row_of(const float *base, uint32_t r, uint64_t ld)
    {
        if (VEC4) return reinterpret_cast<const float *>(reinterpret_cast<const char *>(base) + (uint64_t)r * (uint32_t)(ld * 4));
        return base + r * ld;
    }

    // Even and odd columns are added up separately, two at a time (one instruction each), and then together.
    static __device__ __forceinline__ float dot(const float4 (&x)[V], const float4 (&y)[V])
    {
        uint64_t s = 0;
#pragma unroll
        for (int i = 0; i < V; ++i) {
            s = ptx::fma2(ptx::pack2(x[i].x, x[i].y), ptx::pack2(y[i].x, y[i].y), s);
            s = ptx::fma2(ptx::pack2(x[i].z, x[i].w), ptx::pack2(y[i].z, y[i].w), s);
        }
        const float2 e = ptx::unpack2(s);
        return e.x + e.y;
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
            load(y[u], row_of(a.Y, pr[u].x, a.ldy), c0, a.N, sub);
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

    // 32 nonzeros, lane k's in row `row` and column `col`.  Group g takes nonzeros g * LANES ... one after the other and keeps
    // its row of X in registers (x, loaded by the caller where KEEP): bit k of `turn` says that nonzero k is the first its
    // group sees of its row.  The sums of a group's nonzeros are added over its lanes by halving: at each level a lane hands
    // half of its sums to its partner and keeps the other half, first inside every batch of kFly nonzeros whose rows of Y are in
    // flight together, then over the batches.  That is LANES - 1 shuffles for LANES sums, and a lane is left with the result of
    // nonzero result_of(lane).
    static constexpr int kFly = EACH ? (V == 1 ? 4 : 2) : V == 1 ? LANES : V == 2 ? 4 : 2;  // 16 to 32 registers of Y (EACH: and as many of X)
    static constexpr int kBatches = LANES / kFly;
    static __device__ __forceinline__ uint32_t result_of(int lane)
    {
        const int sub = lane % LANES;
        return (uint32_t)(lane - sub + sub % kBatches * kFly + sub / kBatches);
    }
    template <int CNT> static __device__ __forceinline__ void halve(float *s, int &o, int sub)
    {
#pragma unroll
        for (int left = CNT / 2; left > 0; left /= 2, o /= 2) {
            const bool upper = sub & o;
#pragma unroll
            for (int i = 0; i < left; ++i) {
                const float keep = upper ? s[i + left] : s[i], give = upper ? s[i] : s[i + left];
                s[i] = keep + __shfl_xor_sync(kFull, give, o);
            }
        }
    }
    template <bool KEEP>
    static __device__ __forceinline__ float flat(const SddmmArgs &a, float4 (&x)[V], uint32_t row, unsigned turn, uint32_t col, uint32_t c0, int lane)
    {
        const int sub = lane % LANES, k0 = lane - sub;
        float sums[kBatches];
        int o = LANES / 2;
#pragma unroll
        for (int b = 0; b < kBatches; ++b) {
            float4 y[kFly][V], xs[EACH && !KEEP ? kFly : 1][V];
            float s[kFly];
#pragma unroll
            for (int u = 0; u < kFly; ++u) {
                if constexpr (EACH && !KEEP) load(xs[u], row_of(a.X, __shfl_sync(kFull, row, b * kFly + u, LANES), a.ldx), c0, a.N, sub);
                load(y[u], row_of(a.Y, __shfl_sync(kFull, col, b * kFly + u, LANES), a.ldy), c0, a.N, sub);
            }
#pragma unroll
            for (int u = 0; u < kFly; ++u) {
                const int q = b * kFly + u;
                if constexpr (!KEEP && !EACH)
                    if (turn & (kGroupStarts << q)) {  // the same for every lane
                        const uint32_t r = __shfl_sync(kFull, row, q, LANES);
                        if (turn >> (k0 + q) & 1u) load(x, row_of(a.X, r, a.ldx), c0, a.N, sub);
                    }
                s[u] = dot(EACH && !KEEP ? xs[EACH && !KEEP ? u : 0] : x, y[u]);
            }
            o = LANES / 2;
            halve<kFly>(s, o, sub);
            sums[b] = s[0];
        }
        halve<kBatches>(sums, o, sub);
        return sums[0];
    }
};

// Nonzeros are walked flat, 32 per claim, except where a wide product's rows are not 16-byte aligned: its single-column loads keep a
// warp per row (60 000 x 32 per row N = 101 104 us, flat 130; up to 64 columns flat is faster there too: N = 63 74 -> 72, stencil512
// 143 -> 88.5).
template <int V, bool VEC4> constexpr bool kFlat = VEC4 || V < 3;

template <int LANES, int V, bool VEC4, bool FULL, bool EACH>
__global__ void __launch_bounds__(kTileWarps * 32, kFlat<V, VEC4> ? 4 : 3) sddmm_kernel(SddmmArgs a)
{
    using S = Span<LANES, V, VEC4, FULL, EACH>;
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
                S::load(x, S::row_of(a.X, ck.x, a.ldx), c0, a.N, sub);
                uint2 nxt = __ldg(pairs + min(ck.y + lane, ck.z - 1));  // lanes past the end repeat the last one and store nothing
                for (uint32_t j = ck.y; j < ck.z; j += 32) {
                    const uint2 cur = nxt;
                    if (j + 32 < ck.z) nxt = __ldg(pairs + min(j + 32 + lane, ck.z - 1));
                    const uint32_t n = min(32u, ck.z - j);
                    float v = S::template flat<true>(a, x, 0u, 0u, cur.x, c0, lane);
                    const uint32_t mine = S::result_of(lane);
                    const float scale = __uint_as_float(__shfl_sync(kFull, cur.y, (int)mine));
                    if (mine < n) {
                        if (a.scale) v *= scale;
                        a.out[j + mine] = c0 == 0 ? v : a.out[j + mine] + v;
                    }
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
        if constexpr (kFlat<V, VEC4>) {
            // A warp claims 32 nonzeros at a time whatever their rows; lane i looks the row of the i-th up in the staged row pointers.
            const uint32_t cnt = d.w - d.z;
            for (;;) {
                const uint32_t k0 = tile_claim_rows(ring, s, 32u, lane);
                if (k0 >= cnt) break;
                const uint32_t n = min(32u, cnt - k0), j = d.z + min(k0 + lane, cnt - 1);  // lanes past the end repeat the last nonzero and store nothing
                uint32_t row = d.x, hi = d.y;  // the row with row_ptr[row] <= j < row_ptr[row + 1]
                while (hi - row > 1) {
                    const uint32_t mid = (row + hi) >> 1;
                    if (st.row_ptr[mid - rb] <= j) row = mid; else hi = mid;
                }
                const uint2 cur = st.pairs[j - jb];
                const uint32_t mine = S::result_of(lane);
                const float scale = __uint_as_float(__shfl_sync(kFull, cur.y, (int)mine));
                const uint32_t before = __shfl_up_sync(kFull, row, 1);
                const unsigned turn = __ballot_sync(kFull, row != before) | S::kGroupStarts;
                // the rows of X that a group meets on its way arrive in L1 beside its first loads (R-MAT 2^18 N = 64: 89.6 -> 83.3 us)
                if constexpr (VEC4 && !EACH)
                    if (row != before && lane % LANES) {
                        const float *p = S::row_of(a.X, row, a.ldx);
#pragma unroll
                        for (int i = 0; i < V; ++i) ptx::prefetch_l1(p + 4 * LANES * i);
                    }
                for (uint32_t c0 = 0; c0 < a.N; c0 += S::kCols) {
                    float4 x[V];
                    float v = S::template flat<false>(a, x, row, turn, cur.x, c0, lane);
                    if (mine < n) {
                        float *out = a.out + d.z + k0 + mine;
                        if (a.scale) v *= scale;
                        *out = c0 == 0 ? v : *out + v;
                    }
                }
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
                    S::load(x, S::row_of(a.X, r, a.ldx), c0, a.N, sub);
                    S::items(a, x, pair_at, j1 - j0, a.out + j0, c0, c0 == 0, lane);
                }
            }
        }
        tile_release(ring, src, i, t, lane);
    }
}

template <int LANES, int V, bool VEC4, bool FULL, bool EACH = false> cudaError_t launch_sddmm_t(const SddmmArgs &a, int sm_count, cudaStream_t s)
{
    int per_sm = 0;
    const cudaError_t e = blocks_per_sm<sddmm_kernel<LANES, V, VEC4, FULL, EACH>>(per_sm, kTileWarps * 32);
    if (e != cudaSuccess) return e;
    const uint32_t chunk_blocks = (a.num_chunks + kTileWarps - 1) / kTileWarps;
    uint32_t blocks = a.num_tiles > chunk_blocks ? a.num_tiles : chunk_blocks;
    const uint32_t cap = (uint32_t)(sm_count * per_sm);  // one resident wave
    if (blocks > cap) blocks = cap;
    return launch_overlapped(sddmm_kernel<LANES, V, VEC4, FULL, EACH>, blocks, kTileWarps * 32, 0, s, a);
}
template <int LANES, int V> cudaError_t launch_sddmm_v(const SddmmArgs &a, int sm_count, cudaStream_t s)
{
    if (!a.vec4) return launch_sddmm_t<LANES, V, false, false>(a, sm_count, s);
    // Rows of two or three nonzeros, empty ones apart (a quarter of 400 000 rows with 12 each N = 32 / 64 25.9 / 47.7 us with X loaded each
    // time, 23.1 / 43.4 with X kept): 200 000 x 3 per row N = 16 / 32 / 64 12.8 / 22.9 / 34.0 us with X kept, 11.3 / 19.0 / 32.8 with X
    // loaded each time (before the walk by runs 12.3 / 19.2 / 30.2); 4 per row N = 32 33.2 with X kept, 38.8 before.
    // At 64 columns the walk by runs stays 3 % behind the form before it on the first of these matrices (K = M: 25.9 -> 26.7 us) and is 3 %
    // ahead with 800 000 x 3 of 50 000 columns (77.8 -> 75.3; X kept 27.7 and 74.4, the groups' nonzeros dealt in turn 26.7 and 78.2).
    if constexpr (V <= 2)
        if (a.short_rows)
            return a.N % (4 * V * LANES) == 0 ? launch_sddmm_t<LANES, V, true, true, true>(a, sm_count, s) : launch_sddmm_t<LANES, V, true, false, true>(a, sm_count, s);
    return a.N % (4 * V * LANES) == 0 ? launch_sddmm_t<LANES, V, true, true>(a, sm_count, s) : launch_sddmm_t<LANES, V, true, false>(a, sm_count, s);
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

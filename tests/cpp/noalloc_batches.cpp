// Walks the batches a warp of the no-allocation call makes of a claim of rows (noalloc_rows.hpp; the walk is the kernel's,
// lane by lane) over row pointers of every kind, and checks what the kernel relies on: every position a row reads lies inside
// what its batch has staged, every row is computed once over its own range, and row pointers in order are batched as
// far as the buffer goes.  Needs no GPU.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "../../cutespmm_ae_b200/csrc/noalloc_rows.hpp"

using cutespmm::RowRange;

static int walk(const std::vector<uint32_t> &rp, uint32_t nnz, uint32_t claim, uint32_t split, uint32_t buffer, bool in_order)
{
    const uint32_t M = (uint32_t)rp.size() - 1;
    for (uint32_t first = 0; first < M; first += claim) {
        const uint32_t cnt = std::min(claim, M - first);
        RowRange g[32] = {};
        bool listed[32];
        for (uint32_t i = 0; i < 32; ++i) {
            if (i < cnt) g[i] = cutespmm::row_range(rp[first + i], rp[first + i + 1], nnz);
            if (g[i].j0 > g[i].j1 || g[i].j1 > nnz) return std::printf("row %u: a range outside the arrays\n", first + i), 1;
            listed[i] = g[i].j1 - g[i].j0 > split;
        }
        for (uint32_t i0 = 0; i0 < cnt;) {
            if (listed[i0] || g[i0].j1 - g[i0].j0 > buffer) {  // chunks, or the whole warp on its own range
                ++i0;
                continue;
            }
            uint32_t i1 = i0 + 1;
            while (i1 < 32 && i1 < cnt && !listed[i1] && cutespmm::joins_batch(g[i1 - 1], g[i1], g[i0].j0, buffer)) ++i1;
            const uint32_t staged = g[i1 - 1].j1 - g[i0].j0;
            if (staged > buffer) return std::printf("rows %u..%u: %u nonzeros staged\n", first + i0, first + i1, staged), 1;
            uint32_t start[33];
            for (uint32_t i = i0; i < i1; ++i) start[i] = g[i].j0 - g[i0].j0;
            start[i1] = g[i1 - 1].j1 - g[i0].j0;
            for (uint32_t i = i0; i < i1; ++i) {
                if (start[i + 1] < start[i] || start[i + 1] > staged)
                    return std::printf("row %u reads positions %u..%u of %u staged\n", first + i, start[i], start[i + 1], staged), 1;
                if (g[i0].j0 + start[i] != g[i].j0 || g[i0].j0 + start[i + 1] != g[i].j1)
                    return std::printf("row %u is not computed over its own range\n", first + i), 1;
            }
            if (in_order && i1 < cnt && !listed[i1] && g[i1].j1 - g[i0].j0 <= buffer)
                return std::printf("row %u would have fitted its batch\n", first + i1), 1;
            i0 = i1;
        }
    }
    return 0;
}

int main()
{
    std::mt19937 rng(7);
    int bad = 0;
    for (uint32_t claim : {1u, 2u, 3u, 8u, 32u}) bad |= walk({0, 100, 10, 20}, 300, claim, 128, 256, false);  // ends that go down inside a batch
    for (int round = 0; round < 20000 && !bad; ++round) {
        const uint32_t M = 1 + rng() % 100, claim = 1 + rng() % 32, split = rng() % 2 ? 128 : 0xffffffffu, mean = 1 + rng() % 64;
        std::vector<uint32_t> rp(M + 1, 0u);
        for (uint32_t r = 0; r < M; ++r) rp[r + 1] = rp[r] + rng() % (2 * mean);
        const uint32_t nnz = rp[M];
        bad |= walk(rp, nnz, claim, split, 256, true);
        bad |= walk(rp, nnz / 2, claim, split, 256, true);  // pointers beyond the stated count
        for (uint32_t k = 0; k < 1 + M / 4; ++k) rp[rng() % (M + 1)] = rng() % 3 ? rng() % (nnz + 50) : (uint32_t)rng();
        bad |= walk(rp, nnz, claim, split, 256, false);
    }
    if (!bad) std::printf("ok\n");
    return bad;
}

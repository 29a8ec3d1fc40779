// Which nonzeros a row of the no-allocation call names, and which rows a warp may stage together: the index arithmetic that
// keeps row pointers nobody has checked from leading outside an array.  Plain C++ as well as device code, so that the
// arithmetic can be walked on the CPU over inconsistent row pointers (tests/cpp/noalloc_batches.cpp).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define CUTESPMM_HD __host__ __device__ __forceinline__
#else
#define CUTESPMM_HD inline
#endif

namespace cutespmm {

// Nonzero positions [j0, j1) of a row.
struct RowRange {
    uint32_t j0, j1;
};

// A row's two pointers forced into [0, nnz] and into order: every position an array index is derived from is then below the
// `nnz` the host sized its checks with, whatever the pointers are.
CUTESPMM_HD RowRange row_range(uint32_t begin, uint32_t end, uint32_t nnz)
{
    const uint32_t j0 = begin < nnz ? begin : nnz, j1 = end < nnz ? end : nnz;
    return RowRange{j0, j1 > j0 ? j1 : j0};
}

// Whether row g goes into the batch that starts at position `first` and whose last row so far is `before`.  It has to begin
// where that row ends -- then ends only grow along a batch, so staging [first, end of the last row) holds every row of it, and a
// row's end is the next one's beginning -- and the batch has to fit the buffer.  Row pointers that go down end a batch.
CUTESPMM_HD bool joins_batch(RowRange before, RowRange g, uint32_t first, uint32_t buffer)
{
    return g.j0 == before.j1 && g.j1 - first <= buffer;
}

}  // namespace cutespmm

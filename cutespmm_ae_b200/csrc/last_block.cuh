// Counters that kernels share between launches and leave at zero.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace cutespmm {

// Called by one thread of every block of a launch, after the block's last use of the launch's counters (and a block-wide
// barrier).  True in the block that leaves last: it puts the counters back.  The blocks' shares add up to zero (mod 2^32) for
// any grid, so `balance` is back where it was when a launch has ended, whatever other launches -- of other grids -- ran beside
// it; a launch alone meets zero only when all of its blocks have left.  Launches that overlap may see counters put back
// under them (their results are undefined anyway), but the very last block of all of them always meets zero, so the next
// launch starts from clean counters.  A count modulo the grid's size would keep a remainder then, for good.
__device__ __forceinline__ bool last_block_out(uint32_t *balance)
{
    const uint32_t blocks = gridDim.x * gridDim.y, share = blockIdx.x == 0 && blockIdx.y == 0 ? 1u - blocks : 1u;
    __threadfence();
    return atomicAdd(balance, share) + share == 0u;
}

}  // namespace cutespmm

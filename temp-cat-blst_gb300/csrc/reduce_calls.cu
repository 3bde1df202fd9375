// The reduction's kernels with every field operation a call (no CATMSM_INLINE_*):
// for levels of mostly empty buckets or of few nodes, and for the binary levels (256
// sets of 4096 buckets: 385 us inlined, 378 as calls; 405 and 379 where most are empty).
#include "common.cuh"
#include "reduce.cuh"
#include "catmsm_internal.h"

namespace catmsm {

void reduce_level_calls(const void* inA, const void* inQ, uint32_t m, uint32_t fan_in, uint32_t lg, uint32_t D,
                        bool first, void* outA, void* outQ, cudaStream_t st)
{
    const size_t nodes = (size_t)D * ((m + fan_in - 1) / fan_in);
    k_reduce_level<false><<<div_up(nodes, 128), 128, 0, st>>>((const xyzz*)inA, (const xyzz*)inQ, m, fan_in, lg, D,
                                                              first ? 1 : 0, (xyzz*)outA, (xyzz*)outQ);
}

void reduce_pair_lanes(const void* inA, const void* inQ, uint32_t m, uint32_t D, void* outA, void* outQ,
                       cudaStream_t st)
{
    const size_t nodes = (size_t)D * ((m + 1) / 2);
    k_reduce_pair_lanes<false><<<div_up((nodes + 31) / 32 * 64, 128), 128, 0, st>>>(
        (const xyzz*)inA, (const xyzz*)inQ, m, D, (xyzz*)outA, (xyzz*)outQ);
}

}  // namespace catmsm

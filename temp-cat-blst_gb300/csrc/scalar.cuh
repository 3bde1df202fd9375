// Scalars of the MSM kernels.
#pragma once
#include <cstdint>

namespace catmsm {

// k = the low nbits bits of a little-endian scalar of `stride` bytes
__device__ __forceinline__ void load_scalar(uint32_t* k, const uint8_t* s, uint32_t stride, uint32_t nbits)
{
#pragma unroll
    for (int j = 0; j < 8; j++) k[j] = 0;
    const uint32_t nbytes = (nbits + 7) >> 3;
    if (stride == 32 && (reinterpret_cast<uintptr_t>(s) & 15) == 0) {
        const uint4 a = __ldg(reinterpret_cast<const uint4*>(s));
        const uint4 b = __ldg(reinterpret_cast<const uint4*>(s) + 1);
        k[0] = a.x; k[1] = a.y; k[2] = a.z; k[3] = a.w;
        k[4] = b.x; k[5] = b.y; k[6] = b.z; k[7] = b.w;
    } else if (stride == 16 && (reinterpret_cast<uintptr_t>(s) & 15) == 0) {
        const uint4 a = __ldg(reinterpret_cast<const uint4*>(s));
        k[0] = a.x; k[1] = a.y; k[2] = a.z; k[3] = a.w;
    } else {
        for (uint32_t b = 0; b < nbytes; b++) k[b >> 2] |= (uint32_t)s[b] << (8 * (b & 3));
    }
#pragma unroll
    for (uint32_t j = 0; j < 8; j++) {
        if (nbits <= 32 * j) k[j] = 0;
        else if (nbits < 32 * (j + 1)) k[j] &= (1u << (nbits - 32 * j)) - 1;
    }
}

}  // namespace catmsm

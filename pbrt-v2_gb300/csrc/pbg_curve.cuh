// pbg_curve.cuh -- 3-D Hilbert order of quantised points (ray origins, naive
// triangles).
#pragma once
#include <cstdint>

namespace pbg {

#ifdef __CUDACC__

__device__ __forceinline__ uint32_t spread10(uint32_t v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

// 3-D Hilbert index in transposed form (J. Skilling, "Programming the
// Hilbert curve", AIP Conf. Proc. 707, 2004): the coordinates are rewritten
// in place so that interleaving their bits, as for a Morton code, gives the
// cell's position along the Hilbert curve, whose consecutive cells are
// always face neighbours.
__device__ __forceinline__ void hilbert3(uint32_t x[3], int bits) {
    const uint32_t top = 1u << (bits - 1);
    for (uint32_t q = top; q > 1; q >>= 1) {
        const uint32_t p = q - 1;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (x[a] & q) {
                x[0] ^= p;
            } else {
                const uint32_t t = (x[0] ^ x[a]) & p;
                x[0] ^= t;
                x[a] ^= t;
            }
        }
    }
    x[1] ^= x[0];
    x[2] ^= x[1];
    uint32_t t = 0;
    for (uint32_t q = top; q > 1; q >>= 1)
        if (x[2] & q) t ^= q - 1;
    x[0] ^= t;
    x[1] ^= t;
    x[2] ^= t;
}

#endif  // __CUDACC__

}  // namespace pbg

// Relu and a 2 x 2 max pool on pairs of bf16 channels, and the code that the forward pass leaves for the
// backward one: four bits per channel, the cell of the maximum and 4 when the Relu passes a gradient there.
#pragma once

#include "common.cuh"

namespace ag {
namespace nhwc {

// raw: two channels of the cells (0,0), (0,1), (1,0), (1,1) before the Relu.  Returns the pair's maximum after it;
// code: the two channels' four bits.  Two channels per instruction: one at a time the arithmetic takes longer than the
// memory.
__device__ __forceinline__ uint32_t relu_pool_pair(const uint32_t (&raw)[4], uint32_t &code) {
    const __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);
    __nv_bfloat162 v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = __hmax2(*reinterpret_cast<const __nv_bfloat162 *>(&raw[c]), zero);   // a NaN gives 0
    const __nv_bfloat162 m = __hmax2(__hmax2(v[0], v[1]), __hmax2(v[2], v[3]));
    // the first cell that holds the maximum, and whether the Relu passes its gradient: it does
    // for a positive maximum; a zero one is cell 0's, whose sign decides
    const uint32_t e0 = __heq2_mask(v[0], m), e1 = __heq2_mask(v[1], m), e2 = __heq2_mask(v[2], m);
    const uint32_t pass = __hgt2_mask(m, zero) | __hge2_mask(*reinterpret_cast<const __nv_bfloat162 *>(&raw[0]), zero);
    const uint32_t bit1 = ~e0 & ~e1, bit0 = ~e0 & (e1 | ~e2);
    const uint32_t w = (bit0 & 0x00010001u) | (bit1 & 0x00020002u) | (pass & 0x00040004u);
    code = (w | (w >> 12)) & 0xffu;
    return *reinterpret_cast<const uint32_t *>(&m);
}

}  // namespace nhwc
}  // namespace ag

// A 32-bit value as the sum of three bfloat16 (8 bits of its mantissa each, cut off: exact, and no cut can overflow), for
// products of 32-bit operands on the tensor cores (gemm_f32_tc.cu says what their products leave out).
#pragma once
#include "common.cuh"

namespace fxtc {

// The upper halves of the words returned are the bfloat16.
__device__ __forceinline__ void split3(float x, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = __float_as_uint(x) & 0xffff0000u;
    const float r = x - __uint_as_float(hi);
    mid = __float_as_uint(r) & 0xffff0000u;
    lo = __float_as_uint(r - __uint_as_float(mid));
}
__device__ __forceinline__ uint32_t upper_halves(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }

__device__ __forceinline__ void split3_8(const float* x, uint4& hi, uint4& mid, uint4& lo) {
    uint32_t h[8], m[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) split3(x[i], h[i], m[i], l[i]);
    hi = make_uint4(upper_halves(h[0], h[1]), upper_halves(h[2], h[3]), upper_halves(h[4], h[5]), upper_halves(h[6], h[7]));
    mid = make_uint4(upper_halves(m[0], m[1]), upper_halves(m[2], m[3]), upper_halves(m[4], m[5]), upper_halves(m[6], m[7]));
    lo = make_uint4(upper_halves(l[0], l[1]), upper_halves(l[2], l[3]), upper_halves(l[4], l[5]), upper_halves(l[6], l[7]));
}

}  // namespace fxtc

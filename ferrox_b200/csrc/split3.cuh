// A 32-bit value as the sum of three bfloat16, for products of 32-bit operands on the tensor cores: each is what the ones before it
// left, rounded to nearest, and the third holds the rest exactly (24 bits in three times 8, with signs).  Of a product of two such
// sums, mid.lo, lo.mid and lo.lo are left out: up to 2^-24 of it, of either sign, 2^-27 on average (parts that are cut off instead have
// up to 2^-21, always of the product's sign).  Below 2^-109 the third part, and below 2^-117 the second, no longer have all their
// bits: what is lost of the value is below 2^-133.  What rounds to infinity (from 3.395e38 on) leaves parts that are none.
#pragma once
#include "common.cuh"

namespace fxtc {

// Two values; x in the words' lower halves.
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    auto pack = [&] {
        const __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
        const uint32_t w = *reinterpret_cast<const uint32_t*>(&p);
        x -= __uint_as_float(w << 16);
        y -= __uint_as_float(w & 0xffff0000u);
        return w;
    };
    hi = pack(); mid = pack(); lo = pack();
}

__device__ __forceinline__ void split3_8(const float* x, uint4& hi, uint4& mid, uint4& lo) {
    split3(x[0], x[1], hi.x, mid.x, lo.x);
    split3(x[2], x[3], hi.y, mid.y, lo.y);
    split3(x[4], x[5], hi.z, mid.z, lo.z);
    split3(x[6], x[7], hi.w, mid.w, lo.w);
}

}  // namespace fxtc

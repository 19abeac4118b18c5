// Warp sums of the adjoint kernels.
#pragma once

namespace qg {

// Sums over a warp for FP64 accumulators without the FP64 units (two lanes a clock an SM; a warp of an
// adjoint kernel spent 30 of their instructions, the gradient of 20 steps at 256 x 256 x 3 took 9.30 ms
// with them, 9.13 without).  Pairs of floats carry what a float sum rounds off, 45 bits of the largest
// term and more; operands of a product are scaled by powers of two so that none under- or overflows.
// Infinities and NaN take the FP64 sum.
__device__ __forceinline__ double warp_sum_pair(float h, float l) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float h2 = __shfl_xor_sync(0xffffffffu, h, o), l2 = __shfl_xor_sync(0xffffffffu, l, o);
        const float s = h + h2, b = s - h;
        l += l2 + ((h - (s - b)) + (h2 - b));
        h = s;
    }
    return (double)h + (double)l;
}
__device__ __forceinline__ double warp_sum_f64(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// the sum of v over the warp's lanes, in every lane
__device__ __forceinline__ double warp_total(float v) {
    const unsigned e = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(v))) >> 23;
    return e >= 249 ? warp_sum_f64((double)v) : warp_sum_pair(v, 0.f);  // 32 terms stay below 2^127
}
// the sum of a * b over the warp's lanes, in every lane
__device__ __forceinline__ double warp_dot(float a, float b) {
    const unsigned ea = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(a))) >> 23;
    const unsigned eb = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(b))) >> 23;
    if (ea > 253 || eb > 253) return warp_sum_f64((double)a * (double)b);
    // the largest of each below 2: 2^(127 - e)
    const float x = a * __uint_as_float((254 - ea) << 23), y = b * __uint_as_float((254 - eb) << 23);
    const float h = x * y;
    return warp_sum_pair(h, fmaf(x, y, -h)) * __hiloint2double((int)(ea + eb - 254 + 1023) << 20, 0);
}

}  // namespace qg

// Warp sums of the adjoint kernels.
#pragma once

namespace qg {

// Sums over a warp of four FP64 values at once: lane l gets the total of value l % 4.  FP64 throughout
// (parameter cotangents cancel over the basin, and their terms spread over the whole FP32 range).  The
// first two rounds halve the values a lane holds, so that the four take 6 additions a lane and not 20:
// the FP64 units serve two lanes a clock an SM.  The gradient of 20 steps at 256 x 256 x 3 takes 9.03 ms;
// with a sum for each value 9.30; with products and sums in pairs of FP32 numbers, which lose bits of
// products far below the operands' largest values, 9.07.
__device__ __forceinline__ double warp_sum4(double a, double b, double c, double d) {
    const int lane = threadIdx.x & 31;
    const bool odd = lane & 1, high = lane & 2;
    double ab = odd ? b : a, cd = odd ? d : c;
    ab += __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
    cd += __shfl_xor_sync(0xffffffffu, odd ? c : d, 1);
    double v = high ? cd : ab;
    v += __shfl_xor_sync(0xffffffffu, high ? ab : cd, 2);
#pragma unroll
    for (int o = 4; o < 32; o *= 2) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace qg

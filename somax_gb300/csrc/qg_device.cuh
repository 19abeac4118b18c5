// Device-side PTX helpers shared by the libqgcore kernels: mbarriers with bounded waits,
// TMA tensor copies, programmatic dependent launch.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace qg {

constexpr long long kTimeoutCycles = 4000000000LL;  // ~2 s at 2 GHz: bound of every device wait

__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(su32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: false after kTimeoutCycles or when another role already gave up (*abort).
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, volatile int* abort) {
    if (mbar_try(b, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try(b, parity)) {
        if (abort && *abort) return false;
        if (clock64() - t0 > kTimeoutCycles) {
            if (abort) *abort = 1;
            return false;
        }
    }
    return true;
}
// Bounded wait that ignores the abort flag (draining copies in flight after an abort).
__device__ __forceinline__ bool mbar_drain(uint64_t* b, uint32_t parity) {
    const long long t0 = clock64();
    while (!mbar_try(b, parity))
        if (clock64() - t0 > kTimeoutCycles) return false;
    return true;
}

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

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            su32(dst)),
        "l"((uint64_t)map), "r"(x), "r"(y), "r"(su32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            su32(dst)),
        "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(su32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)map) : "memory");
}

// Programmatic dependent launch.  Every kernel calls pdl_wait() (all prerequisite grids
// complete, their memory visible) before touching data a predecessor writes, and only then
// pdl_launch_dependents(), so at most one launch waits ahead of the running one instead of
// the whole chain cascading onto the SMs.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

}  // namespace qg

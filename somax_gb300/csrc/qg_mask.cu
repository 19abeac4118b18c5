// Device side of the masked-basin inversion: the capacitance correction between the two DST
// solves (host construction and the method in qg_capacitance.cu).
//
// One CTA per (member, mode, block of kCapRows rows of C^-1), a row per warp: sigma_r =
// -sum_j Cinv[r][j] psi_hat[B_j] in FP64, added at B_r to the GEMM operand of the next solve (zero
// there before the first correction: B is land) and to its FP32 copy.  A repeated correction
// removes what the FP32 / split-BF16 solve leaves of psi on B after the first.
//
// Bound: the C^-1 read (8 k^2 bytes per mode) and k^2 FP64 multiply-adds, which the FP64 units take
// about as long for (5 us at k = 1024, three modes); in practice the latency of the reads.  Each lane
// holds kAhead of them in flight and issues the first kAhead before it waits for the solve (C^-1 is a
// constant of the plan).
#include <cuda_bf16.h>

#include "qg_device.cuh"
#include "qg_internal.cuh"

namespace qg {

namespace {

constexpr int NT = 32 * kCapRows;
constexpr int kAhead = 16;  // reads of C^-1 a lane holds in flight

__global__ void __launch_bounds__(NT) k_capacitance(const MemberDev* members, const CapItem* items,
                                                    const float* psi_hat, void* xa, int xa_fmt, float* xq,
                                                    int64_t xplane) {
    extern __shared__ double v[];  // psi_hat of the solve at B
    const CapItem it = items[blockIdx.x];
    const MemberDev& M = members[it.member];
    const int k = M.nb, m = it.mode, Nx = M.Nx;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = it.r0 + warp;
    const double* row = M.cinv + ((size_t)m * k + (r < k ? r : 0)) * k;
    double c[kAhead];
    auto fetch = [&](int j0) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) c[u] = j0 + 32 * u < k ? __ldg(row + j0 + 32 * u) : 0.0;
    };
    fetch(lane);
    const float* ph = psi_hat + M.off_x + (int64_t)m * M.Ny * M.Px;
    pdl_wait();
    pdl_launch_dependents();
    for (int j = threadIdx.x; j < k; j += NT) {
        const int b = M.bidx[j];
        v[j] = (double)ph[(int64_t)(b / Nx) * M.Px + (b % Nx)];
    }
    __syncthreads();
    if (r >= k) return;
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    for (int j0 = lane;;) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (j0 + 32 * u < k) a[u & 3] = fma(c[u], v[j0 + 32 * u], a[u & 3]);
        j0 += 32 * kAhead;
        if (j0 - lane >= k) break;
        fetch(j0);
    }
    double s = (a[0] + a[1]) + (a[2] + a[3]);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) {
        // accumulate: a repeated correction adds to the sources already at B
        const int b = M.bidx[r];
        const int64_t o = M.off_x + ((int64_t)m * M.Ny + b / Nx) * M.Px + (b % Nx);
        if (!xa) {
            // the refinement's residual forms the operand from xq
        } else if (xa_fmt == FMT_F32) {
            float* p = static_cast<float*>(xa);
            p[o] = (float)((double)p[o] - s);
        } else {
            __nv_bfloat16* p = static_cast<__nv_bfloat16*>(xa);
            const double cur = (double)__bfloat162float(p[o]) + (double)__bfloat162float(p[xplane + o]);
            const float sig = (float)(cur - s);
            const __nv_bfloat16 hi = __float2bfloat16_rn(sig);
            p[o] = hi;
            p[xplane + o] = __float2bfloat16_rn(sig - __bfloat162float(hi));
        }
        if (xq) xq[o] = (float)((double)xq[o] - s);
    }
}

}  // namespace

cudaError_t launch_capacitance(const MemberDev* members, const CapItem* items, int n_items, const float* psi_hat,
                               void* xa, int xa_fmt, float* xq, int64_t xplane, size_t smem, cudaStream_t s,
                               bool pdl) {
    if (n_items <= 0) return cudaSuccess;
    return launch_k(k_capacitance, n_items, NT, smem, s, pdl, members, items, psi_hat, xa, xa_fmt, xq, xplane);
}

cudaError_t capacitance_init(size_t max_smem) {
    return cudaFuncSetAttribute(k_capacitance, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_smem);
}

}  // namespace qg

// Row engine of qg_step: a whole Runge-Kutta stage, inversion included, in two FP32 kernels.
//
// The DST-I solve runs x, y, y, x.  Between the two x transforms every column kx of a mode is
// on its own (y transform, divide by ex + ey - lambda, y transform back), and the x transform
// that ends one inversion, the stencil on its psi and the x transform that begins the next
// inversion need only a few neighbouring rows.  So a stage is
//   k_rows  a CTA owns R rows of a member, all layers: inverse x transform of the modes of its
//           rows and one more either side, modes -> layers, Jacobian and the other terms, stage
//           update, layers -> modes, forward x transform of its R rows;
//   k_cols  a CTA owns a few columns kx of one mode: both y transforms and the divide.
// psi, lap(q) and the operand never leave shared memory, and a stage is two launches where the
// pass-by-pass path takes five (six with a Butcher combine).
//
// A transform multiplies the few rows a CTA holds in shared memory by the DST-I matrix with the
// even / odd fold of qg_gemm_simt.cu.  The matrix is stored by quads of k at plan creation
// ([q][n] = S[4q][n] .. S[4q + 3][n], n < ceil(N / 2)) and arrives by bulk copies, in one piece
// when it fits and through a ring of chunks when not; its first copy is on its way before the
// programmatic-dependent-launch wait.
//
// What bounds a transform is the shared-memory data path: every load of a warp returns 4 to 16
// bytes to each of 32 lanes at 128 bytes a cycle, a broadcast read of a row's value as much as a
// read of the matrix.  So a lane takes TN columns (n, n + 32, ...) and RW rows, RW + TN loads for
// RW TN multiply-adds; the warps of a CTA split the columns beyond 32 TN, the rows beyond what a
// lane's registers hold and k, and partial sums over k meet in shared memory.
//
// Every size is a launch argument or a template parameter (layers, rows or columns per CTA, TN):
// with sizes read per member and one kernel for all of them the same launches ran 1500 to 2600
// instructions a warp, most of them index arithmetic and instruction-cache misses (25 us a stage
// at 3 x 130^2).  So the engine takes plans whose members are alike in layers and grid.
//
// A stage measured on GB300, SSP-RK3 (pass by pass with the FP32 passes in brackets): 1 x 66^2
// 7.8 us (12.0), 3 x 130^2 12.0 (17.2), 5 x 142 x 202 19.0 (27.9), 3 x 258^2 24.0 (35.5),
// 1 x 514^2 51 (72), 3 x 514^2 117 (94: the matrix streams, twice the halo work); the split-BF16
// passes take 26 us at 3 x 130^2.  At 3 x 258^2 (cycles of a CTA): loads 3 k, inverse transform
// 10 k, mixes 2 k, lap q 2 k, stencil 4 k, forward transform 7 k; k_cols 2 k + 6.5 k + 6 k + 1 k.
#pragma once

#include "qg_device.cuh"
#include "qg_internal.cuh"

namespace qg {

namespace {

constexpr int kRowWarps = 16;

struct Bars {
    uint64_t full[3];
    int abort;
};

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     su32(dst)),
                 "l"(src), "r"(bytes), "r"(su32(bar))
                 : "memory");
}
// 4 or 16 bytes to shared memory, `bytes` of them read and the rest zero (with 0, src is any valid
// address).
__device__ __forceinline__ void copy4(const float* dst, const float* src, uint32_t bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(su32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy16(const float* dst, const float* src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(su32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The matrix of one axis on its way through shared memory: chunk `seq` of `total` (the matrix
// once per transform when it streams, in one piece when it is resident).
struct Stream {
    const RowAxis& x;
    const float4* g;  // matrix by quads of k (global)
    float4* s;        // slots
    Bars* bars;
    int seq, total;
    __device__ __forceinline__ bool resident() const { return x.nch == 1; }
    __device__ __forceinline__ void issue(int q) {
        const int ch = q >= x.nch ? q - x.nch : q, slot = q % 3;
        const uint32_t bytes = (uint32_t)(min(x.kc, x.quads - ch * x.kc) * x.half) * 16u;
        mbar_expect_tx(&bars->full[slot], bytes);
        bulk_load(s + slot * x.kc * x.half, g + ch * x.kc * x.half, bytes, &bars->full[slot]);
    }
    // thread 0 prepares the barriers and starts the first chunks
    __device__ __forceinline__ void start() {
        if (threadIdx.x != 0) return;
        const int n = min(3, total);
        for (int q = 0; q < n; ++q) mbar_init(&bars->full[q], 1);
        bars->abort = 0;
        mbar_init_fence();
        for (int q = 0; q < n; ++q) issue(q);
    }
    // Before the CTA leaves: a copy that some wait gave up on must not land in a freed CTA.
    __device__ __forceinline__ void leave(int* flags) {
        if (threadIdx.x != 0 || !bars->abort) return;
        for (int q = max(0, total - 3); q < total; ++q) mbar_drain(&bars->full[q % 3], (uint32_t)(q / 3) & 1u);
        if (flags) atomicOr(flags, 2);
    }
};

// t / d for the small quotients of the task loops (RowAxis: d = nc or nw, inv = 65536 / d + 1;
// t d < 65536).
__device__ __forceinline__ int quot(int t, int inv) { return (int)((unsigned)(t * inv) >> 16); }

// The DST of RC rows of X (pitch NP, zero from N to NP): emit(row, n, value) for every output,
// after every thread has read X for the last time.  ks groups of warps share k.  Ends with a CTA
// barrier.  Rows past RC of the last row group are read (they are shared memory of the CTA) and
// dropped.
template <int RC, int TN, class Emit>
__device__ __forceinline__ void transform(Stream& st, const float* X, float* red, int ks, Emit emit) {
    constexpr int RG = row_groups(RC, TN), RW = (RC + RG - 1) / RG;
    const RowAxis& x = st.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g2 = quot(warp, x.ng_inv), ngi = warp - g2 * x.ng;
    const int rg = g2 % RG, kg = g2 / RG;
    const int n0 = ngi * 32 * TN + lane;
    const bool work = kg < ks;
    float2 acc[RW][TN];
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int t = 0; t < TN; ++t) acc[r][t] = make_float2(0.f, 0.f);
    int nn[TN];
#pragma unroll
    for (int t = 0; t < TN; ++t) nn[t] = min(n0 + 32 * t, x.half - 1);
#pragma unroll 1
    for (int ch = 0; ch < x.nch; ++ch) {
        const int slot = st.resident() ? 0 : st.seq % 3;
        mbar_wait(&st.bars->full[slot], st.resident() ? 0u : (uint32_t)(st.seq / 3) & 1u, &st.bars->abort);
        if (work) {
            const int quads = min(x.kc, x.quads - ch * x.kc);
            const float* A = X + rg * RW * x.NP + 4 * ch * x.kc;
            const float4* B = st.s + slot * x.kc * x.half;
#pragma unroll(RW * TN > 16 ? 1 : 2)
            for (int q = kg; q < quads; q += ks) {
                float4 b[TN];
#pragma unroll
                for (int t = 0; t < TN; ++t) b[t] = B[q * x.half + nn[t]];
#pragma unroll
                for (int r = 0; r < RW; ++r) {
                    const float4 a = *reinterpret_cast<const float4*>(A + r * x.NP + 4 * q);
#pragma unroll
                    for (int t = 0; t < TN; ++t)
                        acc[r][t] = __ffma2_rn(make_float2(a.x, a.y), make_float2(b[t].x, b[t].y), acc[r][t]);
#pragma unroll
                    for (int t = 0; t < TN; ++t)
                        acc[r][t] = __ffma2_rn(make_float2(a.z, a.w), make_float2(b[t].z, b[t].w), acc[r][t]);
                }
            }
        }
        if (!st.resident()) {
            __syncthreads();  // the slot is free
            if (threadIdx.x == 0 && st.seq + 3 < st.total) st.issue(st.seq + 3);
            ++st.seq;
        }
    }
    if (ks == 1) {
        __syncthreads();
        if (work) {
#pragma unroll
            for (int r = 0; r < RW; ++r) {
                const int row = rg * RW + r;
                if (row >= RC) break;
#pragma unroll
                for (int t = 0; t < TN; ++t) {
                    const int n = n0 + 32 * t, n2 = x.N - 1 - n;
                    if (n >= x.half) continue;
                    emit(row, n, acc[r][t].x + acc[r][t].y);
                    if (n2 != n) emit(row, n2, acc[r][t].x - acc[r][t].y);
                }
            }
        }
    } else {
        float2* const part = reinterpret_cast<float2*>(red);
        if (work) {
#pragma unroll
            for (int r = 0; r < RW; ++r) {
                const int row = rg * RW + r;
                if (row >= RC) break;
#pragma unroll
                for (int t = 0; t < TN; ++t)
                    if (n0 + 32 * t < x.half) part[(kg * RC + row) * x.half + n0 + 32 * t] = acc[r][t];
            }
        }
        __syncthreads();
        for (int t = warp; t < RC * x.nw; t += kRowWarps) {
            const int r = quot(t, x.nw_inv), c = (t - r * x.nw) * 32 + lane;
            if (c >= x.half) continue;
            const float2* p = part + r * x.half + c;
            float2 v = p[0];
#pragma unroll 4
            for (int g = 1; g < ks; ++g) v = __fadd2_rn(v, p[g * RC * x.half]);
            emit(r, c, v.x + v.y);
            if (x.N - 1 - c != c) emit(r, x.N - 1 - c, v.x - v.y);
        }
    }
    __syncthreads();
}

// Rows ja .. ja + NR - 1 of every layer of a field (`pitch`, `layer`: floats between rows and
// layers) on their way into dst[row][layer][NP]; rows outside the member and columns from N on
// are zero.  wide: 16-byte aligned rows.
template <int NL, int NR>
__device__ __forceinline__ void copy_rows(float* dst, const float* src, int pitch, int64_t layer, bool wide, int ja,
                                          const RowAxis& x, int Ny) {
    const int lane = threadIdx.x & 31;
    for (int w = threadIdx.x >> 5; w < NR * NL; w += kRowWarps) {
        const int r = w / NL, j = ja + r;
        const bool ok = j >= 0 && j < Ny;
        const float* p = ok ? src + (w - r * NL) * layer + (int64_t)j * pitch : src;
        if (wide) {
            for (int i = 4 * lane; i < x.NP; i += 128)
                copy16(dst + w * x.NP + i, p + (ok ? i : 0), ok ? 4u * min(4, x.N - i) : 0u);
        } else {
            for (int i = lane; i < x.NP; i += 32) {
                const bool in = ok && i < x.N;
                copy4(dst + w * x.NP + i, in ? p + i : src, in ? 4u : 0u);
            }
        }
    }
}

// x[row][m] = sum_l C[m][l] x[row][l] in place, NR rows of NL vectors; with `ring0` ring cells
// become zero.
template <int NL, int NR>
__device__ __forceinline__ void mix_rows(float* X, const float* C, int ja, const RowAxis& x, int Ny, bool ring0) {
    float c[NL * NL];
#pragma unroll
    for (int k = 0; k < NL * NL; ++k) c[k] = C[k];
    for (int t = threadIdx.x >> 5; t < NR * x.nc; t += kRowWarps) {
        const int r = quot(t, x.nc_inv), i = (t - r * x.nc) * 32 + (threadIdx.x & 31), j = ja + r;
        if (i >= x.N) continue;
        const bool zero = j < 0 || j >= Ny || (ring0 && (j == 0 || i == 0 || j == Ny - 1 || i == x.N - 1));
        float* p = X + r * NL * x.NP + i;
        float v[NL];
#pragma unroll
        for (int l = 0; l < NL; ++l) v[l] = p[l * x.NP];
#pragma unroll
        for (int m = 0; m < NL; ++m) {
            float s = 0.f;
#pragma unroll
            for (int l = 0; l < NL; ++l) s = fmaf(c[m * NL + l], v[l], s);
            p[m * x.NP] = zero ? 0.f : s;
        }
    }
}

// Rows j0 .. of X[row][layer][NP] to a field; with `ring0` ring cells as zero.
template <int NL, int NR>
__device__ __forceinline__ void store_rows(float* dst, const float* X, int pitch, int64_t layer, int j0,
                                           const RowAxis& x, int Ny, bool ring0) {
    for (int w = threadIdx.x >> 5; w < NR * NL; w += kRowWarps) {
        const int r = w / NL, j = j0 + r;
        if (j >= Ny) break;
        float* p = dst + (w - r * NL) * layer + (int64_t)j * pitch;
        for (int i = threadIdx.x & 31; i < x.N; i += 32) {
            const bool ring = j == 0 || i == 0 || j == Ny - 1 || i == x.N - 1;
            p[i] = ring0 && ring ? 0.f : X[w * x.NP + i];
        }
    }
}

// KIND  kFirst  operand Cl2m q of the rows -> T, and a copy of q
//       kStage  V -> psi -> stencil -> the next stage input and its transform T (and dq)
template <int KIND, int NL, int R, int TN>
__global__ void __launch_bounds__(32 * kRowWarps, 1) k_rows(const __grid_constant__ RowsArgs a) {
    extern __shared__ __align__(16) float sm[];
    __shared__ Bars bars;
    __shared__ float cm[NL * NL], cl[NL * NL], wind[R];
    const RowAxis& x = a.x;
    const int Ny = a.Ny, XP = x.NP, Nx = x.N;
    const MemberDev& M = a.members[blockIdx.y];
    const int j0 = blockIdx.x * R;
    float* const X = sm + a.o_x;      // modes, then psi, of rows j0 - 1 ..
    float* const Q = sm + a.o_q;      // q of rows j0 - 2 ..
    float* const L = sm + a.o_lap;    // lap q of rows j0 - 1 ..; partial sums of the transforms
    float* const O = sm + a.o_op;     // y0, then the stage update, then its modes, of the own rows
    Stream st{x, M.Sx_quad, reinterpret_cast<float4*>(sm + a.o_s), &bars, 0, 0};
    st.total = st.resident() ? 1 : x.nch * (KIND == kStage ? 2 : 1);
    st.start();
    for (int k = threadIdx.x; k < NL * NL; k += 32 * kRowWarps) {
        cm[k] = M.Cm2l[k / NL * kMaxLayers + k % NL];
        cl[k] = M.Cl2m[k / NL * kMaxLayers + k % NL];
    }
    if (KIND == kStage && threadIdx.x < R && j0 + threadIdx.x < Ny) wind[threadIdx.x] = M.F[j0 + threadIdx.x];
    const float idx2 = M.inv_dx2, idy2 = M.inv_dy2, i12 = M.inv_12dxdy, b12 = M.beta_12dx, invH0 = M.invH0;
    const bool psi_ring0 = !M.barotropic;
    const int64_t off_x = M.off_x, off_c = M.off_state, lx = (int64_t)Ny * a.Px, lc = (int64_t)Ny * Nx;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_wait();
    pdl_launch_dependents();
    bool bad = false;

    if constexpr (KIND == kStage) {
        copy_rows<NL, R + 2>(X, a.V + off_x, a.Px, lx, true, j0 - 1, x, Ny);
        copy_rows<NL, R + 4>(Q, a.q + off_x, a.Px, lx, true, j0 - 2, x, Ny);
        if (a.n_k > 0 || a.final_stage || a.a != 0.f) copy_rows<NL, R>(O, a.y0 + off_x, a.Px, lx, true, j0, x, Ny);
        copies_wait();
        __syncthreads();
        // the ring of q reads as zero (the transform's barriers follow)
        for (int w = threadIdx.x; w < (R + 4) * NL; w += 32 * kRowWarps) Q[w * XP] = Q[w * XP + Nx - 1] = 0.f;
        for (int w = warp; w < (R + 4) * NL; w += kRowWarps) {
            const int j = j0 - 2 + w / NL;
            if (j == 0 || j == Ny - 1)
                for (int i = lane; i < Nx; i += 32) Q[w * XP + i] = 0.f;
        }
        transform<(R + 2) * NL, TN>(st, X, L, a.ks_back, [&](int r, int n, float v) { X[r * XP + n] = v; });
        mix_rows<NL, R + 2>(X, cm, j0 - 1, x, Ny, psi_ring0);
        const float* P = a.params + (int64_t)blockIdx.y * QG_NPARAMS;
        const float nu = P[QG_P_NU], kappa = P[QG_P_KAPPA], tau0 = P[QG_P_TAU0] * invH0, nu4 = P[QG_P_NU4];
        const int rowf = NL * XP;  // floats between rows of one layer
        const float* const kp = a.k + off_c;
        float *const dqp = a.dq ? a.dq + off_c : nullptr, *const yp = a.y_next + off_x;
        float chk = 0.f;  // turns NaN on a non-finite value
        for (int t = warp; t < (R + 2) * NL * x.nc; t += kRowWarps) {
            const int w = quot(t, x.nc_inv), i = (t - w * x.nc) * 32 + lane, j = j0 - 1 + w / NL;
            if (i >= Nx) continue;
            const float* c = Q + (w + NL) * XP + i;
            const bool in = j > 0 && j < Ny - 1 && i > 0 && i < Nx - 1;
            L[w * XP + i] = in ? (c[1] - 2.f * c[0] + c[-1]) * idx2 + (c[rowf] - 2.f * c[0] + c[-rowf]) * idy2 : 0.f;
        }
        __syncthreads();
        for (int t = warp; t < R * NL * x.nc; t += kRowWarps) {
            const int w = quot(t, x.nc_inv), i = (t - w * x.nc) * 32 + lane, r = w / NL, l = w - r * NL, j = j0 + r;
            if (i >= XP) continue;
            if (i >= Nx || j >= Ny) {
                O[w * XP + i] = 0.f;
                continue;
            }
            const int ci = (l * Ny + j) * Nx + i, xi = (l * Ny + j) * a.Px + i;  // < 2^31 in a member
            // the earlier stages' derivatives while the stencil computes
            float kv[kMaxButcher - 1];
#pragma unroll
            for (int s = 0; s < kMaxButcher - 1; ++s)
                if (s < a.n_k - 1) kv[s] = kp[s * a.kplane + ci];
            const bool ring = j == 0 || i == 0 || j == Ny - 1 || i == Nx - 1;
            const float wd = l == 0 ? tau0 * wind[r] : 0.f;
            const float* G = Q + (w + 2 * NL) * XP + i;
            float d = wd;
            if (!ring) {
                const float* S = X + (w + NL) * XP + i;
                const float* Lq = L + (w + NL) * XP + i;
                const float fE = S[1], fW = S[-1], fN = S[rowf], fS = S[-rowf];
                const float fNE = S[rowf + 1], fNW = S[rowf - 1], fSE = S[-rowf + 1], fSW = S[-rowf - 1];
                const float gE = G[1], gW = G[-1], gN = G[rowf], gS = G[-rowf];
                const float gNE = G[rowf + 1], gNW = G[rowf - 1], gSE = G[-rowf + 1], gSW = G[-rowf - 1];
                const float jpp = (fE - fW) * (gN - gS) - (fN - fS) * (gE - gW);
                const float jpx = fE * (gNE - gSE) - fW * (gNW - gSW) - fN * (gNE - gNW) + fS * (gSE - gSW);
                const float jxp = gN * (fNE - fNW) - gS * (fSE - fSW) - gE * (fNE - fSE) + gW * (fNW - fSW);
                const float Jb = (4.f * (fE - fW) + (fNE - fNW) + (fSE - fSW)) * b12;
                float v = -((jpp + jpx + jxp) * i12 + Jb) + wd;
                if (l == NL - 1) v += -kappa * ((fE - 2.f * S[0] + fW) * idx2 + (fN - 2.f * S[0] + fS) * idy2);
                v += nu * Lq[0];
                if (nu4 != 0.f)
                    v -= nu4 * ((Lq[1] - 2.f * Lq[0] + Lq[-1]) * idx2 + (Lq[rowf] - 2.f * Lq[0] + Lq[-rowf]) * idy2);
                d = v;
            }
            chk = fmaf(d, 0.f, chk);
            if (dqp) dqp[ci] = d;
            const float y0 = O[w * XP + i];  // when the form reads it
            float yn;
            if (a.n_k > 0) {  // Butcher form: y0 + dt sum_s c_s k_s, the last k this stage's
                float acc = 0.f;
#pragma unroll
                for (int s = 0; s < kMaxButcher - 1; ++s)
                    if (s < a.n_k - 1 && a.coef[s] != 0.f) acc = fmaf(a.coef[s], kv[s], acc);
                if (a.coef_own != 0.f) acc = fmaf(a.coef_own, d, acc);
                yn = y0 + a.dt * acc;
            } else if (ring) {
                yn = a.final_stage ? y0 + a.dt * d : 0.f;  // the ring tendency is the wind's alone
            } else {
                yn = a.b * (G[0] + a.dt * d);
                if (a.a != 0.f) yn += a.a * y0;
            }
            chk = fmaf(yn, 0.f, chk);
            yp[xi] = yn;
            O[w * XP + i] = yn;
        }
        bad = !isfinite(chk);
        __syncthreads();
        mix_rows<NL, R>(O, cl, j0, x, Ny, true);
        __syncthreads();
    } else {
        copy_rows<NL, R>(O, a.q + off_c, Nx, lc, false, j0, x, Ny);
        copies_wait();
        __syncthreads();
        store_rows<NL, R>(a.y_next + off_x, O, a.Px, lx, j0, x, Ny, a.zero_ring != 0);
        __syncthreads();
        mix_rows<NL, R>(O, cl, j0, x, Ny, true);
        __syncthreads();
    }
    transform<R * NL, TN>(st, O, L, a.ks_own, [&](int w, int n, float v) {
        const int r = w / NL, m = w - r * NL;
        if (j0 + r < Ny) a.T[off_x + m * lx + (int64_t)(j0 + r) * a.Px + n] = v;
    });
    if (bad && a.flags) atomicOr(a.flags, 1);
    __syncthreads();
    st.leave(a.flags);
}

// Both y transforms of C columns of one mode around the spectral divide.
template <int C, int TN>
__global__ void __launch_bounds__(32 * kRowWarps, 1) k_cols(const __grid_constant__ ColsArgs a) {
    extern __shared__ __align__(16) float sm[];
    __shared__ Bars bars;
    __shared__ float ex[C];
    const RowAxis& x = a.x;
    const MemberDev& M = a.members[blockIdx.y];
    const int mode = blockIdx.x / a.nblk, i0 = (blockIdx.x - mode * a.nblk) * C;
    float* const X = sm + a.o_x;
    float* const ey = sm + a.o_ey;
    float* const red = sm + a.o_red;
    Stream st{x, M.Sy_quad, reinterpret_cast<float4*>(sm + a.o_s), &bars, 0, 0};
    st.total = st.resident() ? 1 : 2 * x.nch;
    st.start();
    const float* gey = M.ey;
    for (int j = threadIdx.x; j < x.N; j += 32 * kRowWarps) ey[j] = gey[j];
    if (threadIdx.x < C) ex[threadIdx.x] = i0 + threadIdx.x < a.Nx ? M.ex[i0 + threadIdx.x] - M.lam[mode] : 1.f;
    const int64_t base = M.off_x + (int64_t)mode * x.N * a.Px + i0;
    pdl_wait();
    pdl_launch_dependents();
    for (int o = threadIdx.x; o < C * x.NP; o += 32 * kRowWarps) {
        const int j = o / C, k = o - j * C;
        const bool in = j < x.N && i0 + k < a.Nx;
        copy4(X + k * x.NP + j, in ? a.T + base + (int64_t)j * a.Px + k : a.T, in ? 4u : 0u);
    }
    copies_wait();
    __syncthreads();
    transform<C, TN>(st, X, red, a.ks, [&](int k, int n, float v) { X[k * x.NP + n] = v / (ex[k] + ey[n]); });
    transform<C, TN>(st, X, red, a.ks, [&](int k, int n, float v) { X[k * x.NP + n] = v; });
    for (int o = threadIdx.x; o < C * x.N; o += 32 * kRowWarps) {
        const int j = o / C, k = o - j * C;
        if (i0 + k < a.Nx) a.V[base + (int64_t)j * a.Px + k] = X[k * x.NP + j];
    }
    st.leave(a.flags);
}

}  // namespace

// The kernels of one TN (the translation unit's), by (layers, rows) and by columns.
#define QG_ROWS(nl, r, tn) {k_rows<kFirst, nl, r, tn>, k_rows<kStage, nl, r, tn>}
#define QG_NO_ROWS {nullptr, nullptr}
#define QG_ROWS_TABLE(tn)                                                                              \
    const RowsTable kRowsTable##tn = {                                                                 \
        {{QG_ROWS(1, 1, tn), QG_ROWS(1, 2, tn), QG_ROWS(1, 4, tn)},                                    \
         {QG_ROWS(2, 1, tn), QG_ROWS(2, 2, tn), QG_ROWS(2, 4, tn)},                                    \
         {QG_ROWS(3, 1, tn), QG_ROWS(3, 2, tn), QG_ROWS(3, 4, tn)},                                    \
         {QG_ROWS(4, 1, tn), QG_ROWS(4, 2, tn), QG_NO_ROWS},                                           \
         {QG_ROWS(5, 1, tn), QG_ROWS(5, 2, tn), QG_NO_ROWS}},                                          \
        {k_cols<1, tn>, k_cols<2, tn>, k_cols<3, tn>, k_cols<4, tn>, k_cols<6, tn>, k_cols<8, tn>, k_cols<12, tn>, \
         k_cols<16, tn>}};

}  // namespace qg

// Hand-written adjoint (vector-Jacobian product) of the fused RHS and of the PV inversion.
//
// Masked members (land mask): q is read as 0 on land, psi is 0 there and dq = 0 there (wind
// included), lap(q) is zero on land as on the ring; so the cotangent a, qb, psi and M Lf(a)
// are zeroed on land, and so are the cotangents of q and psi at land cells.  The masked
// inversion (two DST solves around the capacitance correction, psi = G x - G E C^-1 R G x with
// G the symmetric solve, C = R G E and R / E the restriction to / extension from the land
// boundary points) is a symmetric map, so the adjoint solve is the same masked inversion.
//
// Forward, per member (baroclinic.py:135-190; B is the optional ring zeroing of q, Z the
// zeroing of the psi ring of the baroclinic model, nu4 the biharmonic extension):
//   qb  = B q,   psi = Z Cm2l L^-1 Cl2m qb
//   dq  = -J(psi, qb) - J(psi, beta y) + nu lap(qb) - nu4 lap(lap qb)
//         + [l = 0] tau0 F / H0 - [l = nl-1] kappa lap(psi)             (J, lap: interior)
// The ring of dq holds the wind term only, so with a = the cotangent g masked to the interior:
//   qb_bar  = -Jg^T(psi; a) + nu Lf(a) - nu4 Lf(M Lf(a))
//   psi_bar = -Jf^T(qb; a) - Jb^T(a) - [l = nl-1] kappa Lf(a)
//   qb_bar += Cl2m^T L^-1 Cm2l^T Z psi_bar
//   q_bar   = B qb_bar
// Jg^T / Jf^T are the transposes of the Arakawa stencil in its second / first argument: for
// every stencil offset o of one argument, the cell b receives a(b - o) times the coefficient
// of that offset at b - o, a sum over the other argument around b - o.  Lf is the 5-point
// Laplacian over the whole array with zeros outside it (the transpose of the interior-only
// Laplacian applied to an interior-masked field) and M masks to the interior.  L^-1 is the
// DST-I solve: S is symmetric and the spectral divide diagonal, so it is self-adjoint and the
// same GEMM passes run it.  The parameter cotangents are the sums of g against the forward
// terms that are linear in nu, kappa, tau0 and nu4.
#include <cuda_bf16.h>

#include <algorithm>

#include "qg_internal.cuh"
#include "qg_stencil_tile.cuh"
#include "qg_warp.cuh"

namespace qg {

namespace {

constexpr int TX = 32, TY = 4, HB = 2;  // tile and halo (the biharmonic reaches two cells)
constexpr int SX = TX + 2 * HB, SY = TY + 2 * HB;
constexpr int NT = 256;

__device__ __forceinline__ bool interior(int j, int i, int Ny, int Nx) {
    return j > 0 && i > 0 && j < Ny - 1 && i < Nx - 1;
}

}  // namespace

// Stencil part of the RHS VJP of members of one layer count: one 32 x 4 tile, every layer, per CTA (128
// threads a layer; blockDim.x = 128 layers).  Writes the direct cotangent of qb (x-row plane `direct`),
// Cm2l^T Z psi_bar as the operand of the adjoint solve (and its FP32 copy for the refinement residual), and
// accumulates the parameter cotangents into `pacc` (double, QG_NPARAMS per member).
//
// Bound: latency on the sizes a gradient is taken of (200 000 cells make 594 CTAs of 384 threads).  The
// layers lie side by side so that their mix is a sum over shared memory; a CTA per layer added them
// up with atomics in a zeroed FP32 plane that another kernel turned into the operand, and a third, of
// sixteen CTAs, summed the wind's cotangent: 41 us a stage at 256 x 256 x 3.  With the finish's sums and
// early starts the gradient of 20 steps there took 9.3 ms, 11.0 before.
//
// A plan of mixed layer counts launches once for each, side by side.  With one launch as wide as the
// deepest member, the CTAs of the others held warps that only waited: a qg_rhs_vjp of 256 members of one,
// three and five layers took 3071 us (2006 so; 2711 with a CTA per layer), of eight small ones 84 (82).
constexpr int kTileThreads = TX * TY, kBox = SX * SY;  // cells of a tile, with its halo
constexpr int kSubX = kTileLX / TX, kSubY = kTileLY / TY;  // CTAs per 64 x 16 tile of the list
constexpr size_t vjp_stencil_smem(int nl) { return (size_t)nl * (4 * kBox + kTileThreads) * sizeof(float); }

__global__ void __launch_bounds__(kTileThreads* kMaxLayers)
    k_vjp_stencil(const MemberDev* members, const StencilTile* tiles, const float* q, int apply_bc, const float* psi,
                  const float* gbar, const float* params, float* direct, void* xa, int xa_fmt, float* xq, int64_t xplane,
                  double* pacc) {
    extern __shared__ float smem[];
    __shared__ MemberDev M;
    __shared__ double red[4][kTileThreads * kMaxLayers / 32];
    const StencilTile t = tiles[blockIdx.x / (kSubX * kSubY)];
    const int part = blockIdx.x % (kSubX * kSubY);
    st::load_member(&M, members + t.member);
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();
    const int Ny = M.Ny, Nx = M.Nx, nl = M.nl;
    const int jt = t.ty * kTileLY + part / kSubX * TY, it = t.tx * kTileLX + part % kSubX * TX;
    if (jt >= Ny || it >= Nx) return;  // all of the CTA
    const int l = threadIdx.x / kTileThreads, c = threadIdx.x % kTileThreads;
    float* sa = smem + (size_t)l * 4 * kBox;             // a = interior-masked cotangent
    float* sq = sa + kBox;                               // qb
    float* sp = sq + kBox;                               // psi (layer, ring zeroed for the baroclinic model)
    float* sm = sp + kBox;                               // M Lf(a)
    float* spb = smem + (size_t)nl * 4 * kBox;           // Z psi_bar of the cells by layer
    const st::CellGeom G(M);
    const float* P = params + (int64_t)t.member * QG_NPARAMS;
    const float nu = P[QG_P_NU], kappa = P[QG_P_KAPPA], nu4 = P[QG_P_NU4];
    const float idx2 = M.inv_dx2, idy2 = M.inv_dy2, i12 = M.inv_12dxdy, b12 = M.beta_12dx;
    const int j0 = jt - HB, i0 = it - HB;
    // the tile and its halo strictly inside a member without land: no rules to apply
    const bool inner = !G.mask && j0 >= 1 && i0 >= 1 && j0 + SY < Ny && i0 + SX < Nx;
    if (inner) {
        const int64_t o0 = G.c(j0, i0) + l * G.lc;
        for (int k = c; k < kBox; k += kTileThreads) {
            const int64_t o = o0 + (k / SX) * Nx + k % SX;
            sa[k] = gbar[o];
            sq[k] = q[o];
            sp[k] = psi[o];
        }
    } else {
        for (int k = c; k < kBox; k += kTileThreads) {
            const int j = j0 + k / SX, i = i0 + k % SX;
            const bool in = j >= 0 && j < Ny && i >= 0 && i < Nx;
            // land of a masked member: dq = 0 there, q is read as 0 and psi is 0
            const bool sea = in && !G.land(j, i), ring = in && G.ring(j, i);
            const int64_t o = G.c(j, i) + l * G.lc;
            sa[k] = sea && !ring ? gbar[o] : 0.f;
            sq[k] = sea && !(apply_bc && ring) ? q[o] : 0.f;
            sp[k] = sea ? psi[o] : 0.f;
        }
    }
    __syncthreads();
    for (int k = c; k < kBox; k += kTileThreads) {
        const int y = k / SX, x = k % SX, j = j0 + y, i = i0 + x;
        float v = 0.f;  // lap(qb) is zero on the ring and on land
        if (y > 0 && x > 0 && y < SY - 1 && x < SX - 1 && (inner || (interior(j, i, Ny, Nx) && !G.land(j, i))))
            v = (sa[k + 1] - 2.f * sa[k] + sa[k - 1]) * idx2 + (sa[k + SX] - 2.f * sa[k] + sa[k - SX]) * idy2;
        sm[k] = v;
    }
    __syncthreads();
    const int j = jt + c / TX, i = it + c % TX, e = (c / TX + HB) * SX + c % TX + HB;
    const bool cell = j < Ny && i < Nx;
    const bool ring = cell && G.ring(j, i), land = cell && G.land(j, i);
    float pb = 0.f, lq = 0.f, lp = 0.f, wind = 0.f;  // of cells that the parameters' terms read
    if (cell) {
        // A(dj, di): a at b + d;  F / Q(cj, ci, dj, di): psi / qb at b + c + d
        auto A = [&](int dj, int di) { return sa[e + dj * SX + di]; };
        auto F = [&](int cj, int ci, int dj, int di) { return sp[e + (cj + dj) * SX + ci + di]; };
        auto Q = [&](int cj, int ci, int dj, int di) { return sq[e + (cj + dj) * SX + ci + di]; };
        // Jg^T: q at offset o of cell c = b - o; coefficient (in psi) of that offset at c
        const float jg =
            A(-1, 0) * ((F(-1, 0, 0, 1) - F(-1, 0, 0, -1)) + (F(-1, 0, 1, 1) - F(-1, 0, 1, -1)))     // N
            - A(1, 0) * ((F(1, 0, 0, 1) - F(1, 0, 0, -1)) + (F(1, 0, -1, 1) - F(1, 0, -1, -1)))      // S
            - A(0, -1) * ((F(0, -1, 1, 0) - F(0, -1, -1, 0)) + (F(0, -1, 1, 1) - F(0, -1, -1, 1)))   // E
            + A(0, 1) * ((F(0, 1, 1, 0) - F(0, 1, -1, 0)) + (F(0, 1, 1, -1) - F(0, 1, -1, -1)))      // W
            + A(-1, -1) * (F(-1, -1, 0, 1) - F(-1, -1, 1, 0))                                        // NE
            + A(1, -1) * (F(1, -1, -1, 0) - F(1, -1, 0, 1))                                          // SE
            + A(-1, 1) * (F(-1, 1, 1, 0) - F(-1, 1, 0, -1))                                          // NW
            + A(1, 1) * (F(1, 1, 0, -1) - F(1, 1, -1, 0));                                           // SW
        // Jf^T: psi at offset o of cell c = b - o; coefficient (in qb) of that offset at c
        const float jf =
            A(0, -1) * ((Q(0, -1, 1, 0) - Q(0, -1, -1, 0)) + (Q(0, -1, 1, 1) - Q(0, -1, -1, 1)))     // E
            - A(0, 1) * ((Q(0, 1, 1, 0) - Q(0, 1, -1, 0)) + (Q(0, 1, 1, -1) - Q(0, 1, -1, -1)))      // W
            - A(-1, 0) * ((Q(-1, 0, 0, 1) - Q(-1, 0, 0, -1)) + (Q(-1, 0, 1, 1) - Q(-1, 0, 1, -1)))   // N
            + A(1, 0) * ((Q(1, 0, 0, 1) - Q(1, 0, 0, -1)) + (Q(1, 0, -1, 1) - Q(1, 0, -1, -1)))      // S
            + A(-1, -1) * (Q(-1, -1, 1, 0) - Q(-1, -1, 0, 1))                                        // NE
            + A(-1, 1) * (Q(-1, 1, 0, -1) - Q(-1, 1, 1, 0))                                          // NW
            + A(1, -1) * (Q(1, -1, 0, 1) - Q(1, -1, -1, 0))                                          // SE
            + A(1, 1) * (Q(1, 1, -1, 0) - Q(1, 1, 0, -1));                                           // SW
        // J(psi, beta y) = beta / (12 dx) [4 (fE - fW) + fNE - fNW + fSE - fSW]
        const float jb = 4.f * (A(0, -1) - A(0, 1)) + (A(-1, -1) - A(-1, 1)) + (A(1, -1) - A(1, 1));
        const float lfa =
            (A(0, 1) - 2.f * A(0, 0) + A(0, -1)) * idx2 + (A(1, 0) - 2.f * A(0, 0) + A(-1, 0)) * idy2;
        const float lfm = (sm[e + 1] - 2.f * sm[e] + sm[e - 1]) * idx2 +
                          (sm[e + SX] - 2.f * sm[e] + sm[e - SX]) * idy2;
        // q and psi of land cells are fixed at 0
        direct[G.x(j, i) + l * G.lx] = land ? 0.f : -jg * i12 + nu * lfa - nu4 * lfm;
        pb = -jf * i12 - jb * b12;
        if (l == nl - 1) pb -= kappa * lfa;
        if ((ring && !M.barotropic) || land) pb = 0.f;
        if (!ring) {
            lq = (Q(0, 0, 0, 1) - 2.f * Q(0, 0, 0, 0) + Q(0, 0, 0, -1)) * idx2 +
                 (Q(0, 0, 1, 0) - 2.f * Q(0, 0, 0, 0) + Q(0, 0, -1, 0)) * idy2;
            if (l == nl - 1)
                lp = (F(0, 0, 0, 1) - 2.f * F(0, 0, 0, 0) + F(0, 0, 0, -1)) * idx2 +
                     (F(0, 0, 1, 0) - 2.f * F(0, 0, 0, 0) + F(0, 0, -1, 0)) * idy2;
        }
        // the wind: every cell of layer 0, ring included; dq = 0 on land
        if (l == 0 && !land) wind = gbar[G.c(j, i)];
    }
    spb[l * kTileThreads + c] = pb;
    // the cotangents: a lap q, -(M Lf(a)) lap q, [bottom] -a lap psi, [top] g F / H0 (a warp is a row)
    const float a0 = cell ? sa[e] : 0.f;
    static_assert(QG_P_NU == 0 && QG_P_KAPPA == 1 && QG_P_TAU0 == 2 && QG_P_NU4 == 3, "the order of the sums");
    const double sum = warp_sum4((double)a0 * lq, l == nl - 1 ? -(double)a0 * lp : 0.0,
                                 l == 0 ? (double)wind * (cell ? M.F[j] : 0.f) * M.invH0 : 0.0,
                                 -(double)(cell ? sm[e] : 0.f) * lq);
    if ((threadIdx.x & 31) < 4) red[threadIdx.x & 31][threadIdx.x >> 5] = sum;
    __syncthreads();
    if (cell) {
        float v = 0.f;
        for (int k = 0; k < nl; ++k) v = fmaf(M.Cm2l[k * kMaxLayers + l], spb[k * kTileThreads + c], v);
        const int64_t o = G.x(j, i) + l * G.lx;
        st::store_plane(xa, xa_fmt, xplane, o, v);
        if (xq) xq[o] = v;
    }
    if (threadIdx.x < 4) {
        double v = 0.0;
        for (int k = 0; k < (int)blockDim.x / 32; ++k) v += red[threadIdx.x][k];
        atomicAdd(&pacc[QG_NPARAMS * t.member + threadIdx.x], v);
    }
}

// The operand of the adjoint solve of the inversion's VJP, Cm2l^T Z psi_bar of a caller-packed layer
// cotangent (plus its FP32 copy for the refinement residual).
__global__ void __launch_bounds__(NT, 4) k_vjp_operand(const MemberDev* members, const StencilTile* tiles, int parts,
                                                    const float* psi_bar, void* xa, int xa_fmt,
                                                    float* xq, int64_t xplane) {
    __shared__ MemberDev M;
    const StencilTile t = tiles[blockIdx.x / (unsigned)parts];
    st::load_member(&M, members + t.member);
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();
    const st::CellGeom G(M);
    st::with_layers(M.nl, [&](auto n) {
        constexpr int NL = decltype(n)::value;
        const st::Mix<NL, true> C(M.Cm2l);
        const bool keep_ring = M.barotropic;
        st::walk_cells<NL, NL <= 4 ? 4 : 2>(
            G, t, parts,
            [&](int j, int i, float(&x)[NL]) {
                const int64_t c = G.c(j, i);
#pragma unroll
                for (int l = 0; l < NL; ++l) x[l] = psi_bar[c + l * G.lc];
            },
            [&](int j, int i, float(&x)[NL]) {
                const bool zero = (!keep_ring && G.ring(j, i)) || G.land(j, i);
                const int64_t o = G.x(j, i);
#pragma unroll
                for (int m = 0; m < NL; ++m) {
                    const float v = zero ? 0.f : C.row(m, x);
                    st::store_plane(xa, xa_fmt, xplane, o + m * G.lx, v);
                    if (xq) xq[o + m * G.lx] = v;
                }
            });
    });
}

// Linear combinations over packed fields for the Runge-Kutta step's adjoint: n_terms fields x_j or y_j
// with coefficients c_j.
struct LinComb {
    const float* x[kMaxButcher];
    float* y[kMaxButcher];
    float c[kMaxButcher];
    int n_terms;
};

// v = B (direct + Cl2m^T x_bar) in caller packing, x_bar the adjoint solve's output: q_bar = v, or
// (ADD, the step's adjoint) q_bar += v and y_j += c_j v, which a separate pass over v did before.
template <bool ADD>
__global__ void __launch_bounds__(NT, 4) k_vjp_finish(const MemberDev* members, const StencilTile* tiles, int parts,
                                                   const float* direct, const float* xbar, int apply_bc, float* qbar,
                                                   LinComb lc) {
    __shared__ MemberDev M;
    const StencilTile t = tiles[blockIdx.x / (unsigned)parts];
    st::load_member(&M, members + t.member);
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();
    const st::CellGeom G(M);
    st::with_layers(M.nl, [&](auto n) {
        constexpr int NL = decltype(n)::value;
        const st::Mix<NL, true> C(M.Cl2m);
        st::walk_cells<2 * NL, ADD ? 1 : NL <= 2 ? 4 : NL <= 4 ? 2 : 1>(
            G, t, parts,
            [&](int j, int i, float(&x)[2 * NL]) {
                const int64_t o = G.x(j, i);
#pragma unroll
                for (int l = 0; l < NL; ++l) {
                    x[l] = xbar[o + l * G.lx];
                    x[NL + l] = direct ? direct[o + l * G.lx] : 0.f;
                }
            },
            [&](int j, int i, float(&x)[2 * NL]) {
                // q of the ring (under the BC) and of land cells is not read by the forward
                const bool zero = (apply_bc && G.ring(j, i)) || G.land(j, i);
                const int64_t c = G.c(j, i);
                float v[NL];
#pragma unroll
                for (int l = 0; l < NL; ++l) v[l] = zero ? 0.f : C.row(l, x, x[NL + l]);
                if constexpr (ADD) {
                    // the sums' old values of every layer ahead of the stores
                    float old[NL];
#pragma unroll
                    for (int l = 0; l < NL; ++l) old[l] = qbar[c + l * G.lc];
#pragma unroll
                    for (int k = 0; k < kMaxButcher; ++k) {
                        float kb[NL];
                        const bool term = k < lc.n_terms;
#pragma unroll
                        for (int l = 0; l < NL; ++l) kb[l] = term ? lc.y[k][c + l * G.lc] : 0.f;
#pragma unroll
                        for (int l = 0; l < NL; ++l)
                            if (term) lc.y[k][c + l * G.lc] = fmaf(lc.c[k], v[l], kb[l]);
                    }
#pragma unroll
                    for (int l = 0; l < NL; ++l) v[l] += old[l];
                }
#pragma unroll
                for (int l = 0; l < NL; ++l) qbar[c + l * G.lc] = v[l];
            });
    });
}

__global__ void k_vjp_params(const double* __restrict__ pacc, int n, float* __restrict__ pbar) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) pbar[k] = (float)pacc[k];
}

cudaError_t launch_vjp_stencil(const VjpArgs& v, int nl, const StencilTile* tiles, int n, cudaStream_t s, bool pdl) {
    return launch_k(k_vjp_stencil, n * kSubX * kSubY, kTileThreads * nl, vjp_stencil_smem(nl), s, pdl, v.members, tiles,
                    v.q, v.apply_bc, v.psi, v.gbar, v.params, v.direct, v.xa, v.xa_fmt, v.xq, v.xplane, v.pacc);
}

cudaError_t launch_vjp_operand(const VjpArgs& v, const float* psi_bar, cudaStream_t s) {
    const int parts = cell_parts(v.n_cells);
    return launch_k(k_vjp_operand, v.n_cells * parts, NT, 0, s, v.pdl, v.members, v.cells, parts, psi_bar, v.xa, v.xa_fmt,
                    v.xq, v.xplane);
}

cudaError_t launch_vjp_finish(const VjpArgs& v, const float* xbar, float* qbar, cudaStream_t s) {
    const int parts = cell_parts(v.n_cells);
    return launch_k(k_vjp_finish<false>, v.n_cells * parts, NT, 0, s, v.pdl, v.members, v.cells, parts, v.direct, xbar,
                    v.apply_bc, qbar, LinComb{});
}

// ybar += v and kbar[j] += c[j] v (j < n_terms) with v as launch_vjp_finish's
cudaError_t launch_vjp_scatter(const VjpArgs& v, const float* xbar, float* ybar, float* const* kbar, const float* c,
                               int n_terms, cudaStream_t s) {
    LinComb lc{};
    lc.n_terms = n_terms;
    for (int j = 0; j < n_terms; ++j) {
        lc.y[j] = kbar[j];
        lc.c[j] = c[j];
    }
    const int parts = cell_parts(v.n_cells);
    return launch_k(k_vjp_finish<true>, v.n_cells * parts, NT, 0, s, v.pdl, v.members, v.cells, parts, v.direct, xbar,
                    v.apply_bc, ybar, lc);
}

// out = base + sum_j c_j x_j (the stage inputs), n floats
__global__ void __launch_bounds__(NT) k_lincomb(float* out, const float* base, LinComb lc, int64_t n) {
    pdl_wait();
    pdl_launch_dependents();
    const int64_t nth = (int64_t)gridDim.x * NT;
    for (int64_t t = blockIdx.x * (int64_t)NT + threadIdx.x; t < n; t += nth) {
        float v = base[t];
#pragma unroll
        for (int j = 0; j < kMaxButcher; ++j)
            if (j < lc.n_terms) v = fmaf(lc.c[j], lc.x[j][t], v);
        out[t] = v;
    }
}

// y_j = c_j g for every stage j (the cotangents of the stage derivatives at the step's end), and the
// n_acc parameter sums to zero (a memset would keep the next launch from starting early).
__global__ void __launch_bounds__(NT) k_fanout(const float* g, LinComb lc, int64_t n, double* acc, int n_acc) {
    pdl_wait();
    pdl_launch_dependents();
    const int64_t nth = (int64_t)gridDim.x * NT, t0 = blockIdx.x * (int64_t)NT + threadIdx.x;
    for (int64_t t = t0; t < n_acc; t += nth) acc[t] = 0.0;
    for (int64_t t = t0; t < n; t += nth) {
        const float v = g[t];
#pragma unroll
        for (int j = 0; j < kMaxButcher; ++j)
            if (j < lc.n_terms) lc.y[j][t] = lc.c[j] * v;
    }
}

namespace {
int lincomb_grid(int64_t n) { return (int)std::min<int64_t>(8192, std::max<int64_t>(1, (n + 255) / 256)); }
}  // namespace

cudaError_t launch_lincomb(float* out, const float* base, const float* const* x, const float* c, int n_terms,
                           int64_t n, cudaStream_t s, bool pdl) {
    LinComb lc{};
    lc.n_terms = n_terms;
    for (int j = 0; j < n_terms; ++j) {
        lc.x[j] = x[j];
        lc.c[j] = c[j];
    }
    return launch_k(k_lincomb, lincomb_grid(n), NT, 0, s, pdl, out, base, lc, n);
}

cudaError_t launch_fanout(const float* g, float* const* out, const float* c, int n_terms, int64_t n, double* acc,
                          int n_acc, cudaStream_t s, bool pdl) {
    LinComb lc{};
    lc.n_terms = n_terms;
    for (int j = 0; j < n_terms; ++j) {
        lc.y[j] = out[j];
        lc.c[j] = c[j];
    }
    return launch_k(k_fanout, lincomb_grid(n), NT, 0, s, pdl, g, lc, n, acc, n_acc);
}

cudaError_t launch_vjp_params_only(const VjpArgs& v, float* pbar, cudaStream_t s) {
    const int n = v.n_members * QG_NPARAMS;
    k_vjp_params<<<(n + 127) / 128, 128, 0, s>>>(v.pacc, n, pbar);
    return cudaGetLastError();
}

}  // namespace qg

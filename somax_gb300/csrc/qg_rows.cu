// Host side of the FP32 row engine (kernels: qg_rows.cuh): layouts, kernel tables, launches.
#include <algorithm>

#include "qg_internal.cuh"

namespace qg {

extern const RowsTable kRowsTable1, kRowsTable2, kRowsTable3, kRowsTable4, kRowsTable5;

namespace {

constexpr size_t kSmemBudget = 226 * 1024;
constexpr int kWarps = 16;
constexpr int kRowOptions[3] = {1, 2, 4};                       // rows per CTA of k_rows
constexpr int kColOptions[8] = {1, 2, 3, 4, 6, 8, 12, 16};      // columns per CTA of k_cols

const RowsTable& table(int tn) {
    static const RowsTable* const t[5] = {&kRowsTable1, &kRowsTable2, &kRowsTable3, &kRowsTable4, &kRowsTable5};
    return *t[tn - 1];
}

int up(int v, int m) { return (v + m - 1) / m * m; }

// Geometry of one axis of N points and the cut of its matrix for `bytes` of shared memory: in one
// piece, or in chunks of kc quads of k through three slots.  False: neither fits.
bool axis_for(int N, size_t bytes, RowAxis* a) {
    a->N = N;
    a->half = (N + 1) / 2;
    a->NP = up(N, 4);
    a->quads = a->NP / 4;
    a->nw = (a->half + 31) / 32;
    a->nc = (a->NP + 31) / 32;
    a->ng = (a->nw + 4) / 5;
    a->tn = (a->nw + a->ng - 1) / a->ng;
    if (4 * a->ng > kWarps) return false;
    a->nw_inv = 65536 / a->nw + 1;
    a->nc_inv = 65536 / a->nc + 1;
    a->ng_inv = 65536 / a->ng + 1;
    const size_t quad = (size_t)a->half * 16;
    if (a->quads * quad <= bytes) {
        a->kc = a->quads;
        a->nch = 1;
        return true;
    }
    a->kc = std::min(16, (int)(bytes / (3 * quad)));
    if (a->kc < 2) return false;
    a->nch = (a->quads + a->kc - 1) / a->kc;
    return true;
}
size_t axis_bytes(const RowAxis& a) { return (size_t)(a.nch == 1 ? a.quads : 3 * a.kc) * a.half * 16; }
// Warp groups over k of a transform of `rows` rows: at most `most` (more groups add more partial
// sums than they save), and the floats of their partial sums.
int k_groups(const RowAxis& a, int rows, int most) {
    return std::max(1, std::min(most, kWarps / (a.ng * row_groups(rows, a.tn))));
}
int red_floats(const RowAxis& a, int rows, int ks) { return ks > 1 ? up(ks * rows * a.half * 2, 4) : 0; }

// The layouts try 8 k groups, then fewer, until the matrix fits beside the partial sums in one
// piece; failing that, 2 groups and the matrix in chunks.
bool rows_layout(int nl, int R, int Nx, RowsArgs* a) {
    for (int most : {8, 4, 2}) {
        RowAxis& x = a->x;
        if (!axis_for(Nx, (size_t)1 << 30, &x)) return false;
        const int n = nl * x.NP;
        a->ks_back = k_groups(x, (R + 2) * nl, most);
        a->o_x = 0;
        a->o_q = a->o_x + (R + 2) * n;
        a->o_lap = a->o_q + (R + 4) * n;
        const int lap = std::max((R + 2) * n, red_floats(x, (R + 2) * nl, a->ks_back));
        a->ks_own = k_groups(x, R * nl, 8);  // as many as the same space holds
        while (red_floats(x, R * nl, a->ks_own) > lap) --a->ks_own;
        a->o_op = a->o_lap + lap;
        a->o_s = a->o_op + R * n;
        const size_t fixed = (size_t)a->o_s * 4;
        if (fixed >= kSmemBudget || !axis_for(Nx, kSmemBudget - fixed, &x) || (x.nch > 1 && most > 2)) continue;
        a->smem = fixed + axis_bytes(x);
        a->rows = R;
        a->layers = nl;
        return true;
    }
    return false;
}
bool cols_layout(int c, int Ny, ColsArgs* a) {
    for (int most : {8, 4, 2}) {
        RowAxis& x = a->x;
        if (!axis_for(Ny, (size_t)1 << 30, &x)) return false;
        a->ks = k_groups(x, c, most);
        a->o_x = 0;
        a->o_ey = a->o_x + c * x.NP;
        a->o_red = a->o_ey + x.NP;
        a->o_s = a->o_red + red_floats(x, c, a->ks);
        const size_t fixed = (size_t)a->o_s * 4;
        if (fixed >= kSmemBudget || !axis_for(Ny, kSmemBudget - fixed, &x) || (x.nch > 1 && most > 2)) continue;
        a->smem = fixed + axis_bytes(x);
        a->cols = c;
        return true;
    }
    return false;
}

int row_option(int R) { return R == 4 ? 2 : R - 1; }
RowsKernel rows_kernel(int kind, const RowsArgs& a) {
    if (kind < 0 || kind > 1 || a.layers < 1 || a.layers > kRowLayers || row_option(a.rows) < 0 || row_option(a.rows) > 2)
        return nullptr;
    return table(a.x.tn).rows[a.layers - 1][row_option(a.rows)][kind];
}
ColsKernel cols_kernel(const ColsArgs& a) {
    for (int k = 0; k < 8; ++k)
        if (kColOptions[k] == a.cols) return table(a.x.tn).cols[k];
    return nullptr;
}

template <class K, class A>
cudaError_t launch_grid(K kernel, dim3 grid, const A& a, cudaStream_t s, bool pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(32 * kWarps);
    cfg.dynamicSmemBytes = a.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

}  // namespace

int rows_quad_floats(int N) { return up(N, 4) * ((N + 1) / 2); }

// The matrix S (N x N, pitch ld) by quads of k: out[q][n] = (S[4 q][n], .. S[4 q + 3][n]),
// n < ceil(N / 2), zero past the last k.
void rows_quad_matrix(const float* S, int N, int ld, float* out) {
    const int half = (N + 1) / 2;
    for (int k = 0; k < up(N, 4); ++k)
        for (int n = 0; n < half; ++n) out[((size_t)(k / 4) * half + n) * 4 + k % 4] = k < N ? S[(size_t)k * ld + n] : 0.f;
}

// Layout of the two launches for n_members alike members: the fewest rows (columns) per CTA that
// need no second wave of CTAs, or the most that fit.
bool rows_plan(int nl, int Ny, int Nx, int n_members, int n_sm, RowsArgs* r, ColsArgs* c) {
    if (nl < 1 || nl > kRowLayers) return false;
    int best = 0;
    for (int k = 0; k < 3; ++k) {
        RowsArgs t = *r;
        if (!rows_layout(nl, kRowOptions[k], Nx, &t) || !table(t.x.tn).rows[nl - 1][k][0]) break;
        *r = t;
        best = kRowOptions[k];
        if ((int64_t)((Ny + best - 1) / best) * n_members <= n_sm) break;
    }
    if (!best) return false;
    r->Ny = Ny;
    r->bands = (Ny + best - 1) / best;
    best = 0;
    for (int k = 0; k < 8; ++k) {
        ColsArgs t = *c;
        if (!cols_layout(kColOptions[k], Ny, &t)) break;
        *c = t;
        best = kColOptions[k];
        if ((int64_t)((Nx + best - 1) / best) * nl * n_members <= n_sm) break;
    }
    if (!best) return false;
    c->Nx = Nx;
    c->nblk = (Nx + best - 1) / best;
    c->layers = nl;
    return true;
}

// Whether a plan that is not timed steps with the row engine: by the CTAs of k_rows (an SM holds one) and
// the multiply-adds of one (its rows' two transforms).  In one wave the engine loses only where the
// streamed matrix and the halo rows weigh; further waves each load the matrix again, which one-layer
// members bear longest, and tiny members not at all.  Measured over 334 plans (64^2 to 1000^2 and oblong,
// 1 to 5 layers, 1 to 128 alike members, four SSP-RK3 steps; engine / FP32 passes): 3 x 448^2 0.99 / 1.02
// ms, 3 x 514^2 1.45 / 1.17, 3 x 1002^2 14.9 / 5.0; members of 1 x 130^2: 16 0.45 / 0.53, 32 0.79 / 0.65;
// of 3 x 130^2: 8 0.51 / 0.52, 16 0.88 / 0.70; of 3 x 66^2: 8 0.20 / 0.30, 16 0.37 / 0.34.  Where the rule
// takes the engine it loses 4 % at most; where it does not, the engine gains 22 % at most.
bool rows_pay(const RowsArgs& r, int n_members, int n_sm) {
    const int64_t ctas = (int64_t)r.bands * n_members;
    const int64_t work = (int64_t)(2 * r.rows + 2) * r.layers * r.x.half * r.x.NP;
    if (ctas <= n_sm) return work <= 3200000;
    if (r.layers == 1) return 2 * ctas <= 7 * n_sm && work <= 1050000;
    return ctas <= 2 * n_sm && r.layers <= 4 && r.x.nch == 1 && work >= 70000;
}

// Allow the plan's kernels their shared memory (on the current device).
cudaError_t rows_init(const RowsArgs& r, const ColsArgs& c) {
    cudaError_t e = cudaFuncSetAttribute(cols_kernel(c), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget);
    for (int kind = 0; kind < 2 && !e; ++kind)
        e = cudaFuncSetAttribute(rows_kernel(kind, r), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget);
    return e;
}
cudaError_t launch_rows(int kind, const RowsArgs& a, int n_members, cudaStream_t s, bool pdl) {
    const RowsKernel k = rows_kernel(kind, a);
    return k ? launch_grid(k, dim3(a.bands, n_members), a, s, pdl) : cudaErrorInvalidValue;
}
cudaError_t launch_cols(const ColsArgs& a, int n_members, cudaStream_t s, bool pdl) {
    const ColsKernel k = cols_kernel(a);
    return k ? launch_grid(k, dim3(a.nblk * a.layers, n_members), a, s, pdl) : cudaErrorInvalidValue;
}

}  // namespace qg

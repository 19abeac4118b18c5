// FP32 DST-I passes on the CUDA cores (the plans' default precision, and qg_invert_static).
//
// Each pass is C = A S with S the symmetric orthonormal DST-I matrix of the contracted axis,
// stored transposed.  S[k][N-1-n] = (-1)^k S[k][n], so with the even and the odd k of a row
// summed apart,
//     E[n] = sum_{k even} A[k] S[k][n],  O[n] = sum_{k odd} A[k] S[k][n]   (n < ceil(N / 2)),
//     C[n] = E[n] + O[n],                C[N-1-n] = E[n] - O[n]:
// half the multiply-adds of the plain product, and half the terms in each FP32 sum.  The pairs
// (A[k], A[k+1]) and (S[n][k], S[n][k+1]), k even, are neighbours in memory and become the two
// halves of one packed FP32x2 multiply-add whose accumulator is (E, O).
//
// A CTA forms BM rows x BN of those columns (2 BN of C); 16 threads run along the rows (row
// r0 + 16 i, so that 16 lanes store 64 consecutive bytes of a transposed output row) and CT
// along the columns.  Pairs travel to shared memory by 8-byte cp.async, which transposes them
// on the way ([k pair][row], odd pitch: neither the copies nor the reads conflict), through a
// ring of STAGES slots; the columns' pairs do not depend on the previous kernel, so the first
// slots' are under way before the programmatic-dependent-launch wait.
//
// Bound: FP32 issue on large members, L2 latency and the launch on small ones.  The shapes
// differ in work per thread (multiply-adds per shared-memory read) against CTAs in flight.
#include "qg_device.cuh"
#include "qg_internal.cuh"

namespace qg {

namespace {

constexpr int kRowThreads = 16;

template <int TM_, int TN_, int CT_, int BKP_, int STAGES_>
struct Shape {
    static constexpr int TM = TM_, TN = TN_, CT = CT_, BKP = BKP_, STAGES = STAGES_;
    static constexpr int BM = kRowThreads * TM, BN = CT * TN, NT = kRowThreads * CT;
    static constexpr int PA = BM + 1, PB = BN | 1;  // odd pitches (in pairs)
    static constexpr int SLOT = BKP * (PA + PB);
    static constexpr size_t SMEM = (size_t)STAGES * SLOT * sizeof(float2);
};

using Shape0 = Shape<4, 6, 8, 16, 3>;  // 64 x 48
using Shape1 = Shape<4, 3, 8, 16, 4>;  // 64 x 24
using Shape2 = Shape<2, 3, 8, 16, 5>;  // 32 x 24
using Shape3 = Shape<1, 1, 8, 16, 6>;  // 16 x 8

struct PassGeom {
    int Mb, K, Mtot, lda, ldo;
    const float* A;
    const float* B;
    float* C;
};

__device__ __forceinline__ PassGeom pass_geom(const MemberDev& M, int pass, const void* A, void* C) {
    PassGeom g;
    const bool xin = pass_xin(pass);  // A in x-row planes, C (transposed) in y-row planes
    g.Mb = xin ? M.Ny : M.Nx;
    g.K = xin ? M.Nx : M.Ny;
    g.Mtot = M.nl * g.Mb;
    g.lda = xin ? M.Px : M.Py;
    g.ldo = xin ? M.Py : M.Px;
    g.A = static_cast<const float*>(A) + (xin ? M.off_x : M.off_y);
    g.B = xin ? M.Sx : M.Sy;
    g.C = static_cast<float*>(C) + (xin ? M.off_y : M.off_x);
    return g;
}

// One pair to shared memory: `bytes` (0, 4 or 8) read, the rest zero.
__device__ __forceinline__ void copy_pair(const float2* dst, const float* src, uint32_t bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(su32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Pairs [kb, kb + BKP) of rows row0 .. row0 + R - 1 of a K-contiguous operand (pitch ld) into
// dst[pair][row] (pitch P); rows from `rows` on and elements from K on are zero, not read.
template <class S, int R, int P>
__device__ __forceinline__ void copy_rows(float2* dst, const float* src, int ld, int row0, int rows, int kb, int K) {
    constexpr int STEP = S::NT / S::BKP;
    const int kp = threadIdx.x % S::BKP, k = 2 * (kb + kp);
    const uint32_t kbytes = k + 1 < K ? 8u : (k < K ? 4u : 0u);
#pragma unroll
    for (int i = 0; i < (R + STEP - 1) / STEP; ++i) {
        const int r = threadIdx.x / S::BKP + i * STEP;
        if (R % STEP != 0 && r >= R) break;
        const bool ok = row0 + r < rows && kbytes != 0u;
        copy_pair(dst + kp * P + r, ok ? src + (int64_t)(row0 + r) * ld + k : src, ok ? kbytes : 0u);
    }
}

template <class S>
__device__ __forceinline__ void mul_pairs(float2 (&acc)[S::TM][S::TN], const float2* As, const float2* Bs) {
    float2 a[S::TM], b[S::TN];
#pragma unroll
    for (int i = 0; i < S::TM; ++i) a[i] = As[kRowThreads * i];
#pragma unroll
    for (int j = 0; j < S::TN; ++j) b[j] = Bs[S::CT * j];
#pragma unroll
    for (int i = 0; i < S::TM; ++i)
#pragma unroll
        for (int j = 0; j < S::TN; ++j) acc[i][j] = __ffma2_rn(a[i], b[j], acc[i][j]);
}

template <int PASS, class S>
__global__ void __launch_bounds__(S::NT) k_gemm_simt(GemmArgs ga) {
    extern __shared__ __align__(16) float2 ring[];
    const GemmTile t = ga.tiles[blockIdx.x];
    const MemberDev& M = ga.members[t.member];
    const PassGeom g = pass_geom(M, PASS, ga.A, ga.C);
    const int m0 = t.mt * S::BM, n0 = t.nt * S::BN;
    const int half = (g.K + 1) / 2;  // columns formed, and pairs contracted
    const int nkb = (half + S::BKP - 1) / S::BKP;
    float2* const ringB = ring + S::BKP * S::PA;
#pragma unroll
    for (int s = 0; s < S::STAGES - 1; ++s)
        if (s < nkb) copy_rows<S, S::BN, S::PB>(ringB + s * S::SLOT, g.B, g.lda, n0, half, s * S::BKP, g.K);
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll
    for (int s = 0; s < S::STAGES - 1; ++s) {
        if (s < nkb) copy_rows<S, S::BM, S::PA>(ring + s * S::SLOT, g.A, g.lda, m0, g.Mtot, s * S::BKP, g.K);
        copy_commit();
    }
    const int mr = threadIdx.x % kRowThreads, nc = threadIdx.x / kRowThreads;
    float2 acc[S::TM][S::TN];
#pragma unroll
    for (int i = 0; i < S::TM; ++i)
#pragma unroll
        for (int j = 0; j < S::TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
    int slot = 0, fill = S::STAGES - 1;
#pragma unroll 1
    for (int kt = 0; kt < nkb; ++kt) {
        copy_wait<S::STAGES - 2>();
        __syncthreads();  // slot kt has landed for every thread; slot kt - 1 is free
        if (kt + S::STAGES - 1 < nkb) {
            const int kb = (kt + S::STAGES - 1) * S::BKP;
            copy_rows<S, S::BM, S::PA>(ring + fill * S::SLOT, g.A, g.lda, m0, g.Mtot, kb, g.K);
            copy_rows<S, S::BN, S::PB>(ringB + fill * S::SLOT, g.B, g.lda, n0, half, kb, g.K);
        }
        copy_commit();
        const float2* As = ring + slot * S::SLOT + mr;
        const float2* Bs = ringB + slot * S::SLOT + nc;
        const int kn = half - kt * S::BKP;
        if (kn >= S::BKP) {
#pragma unroll
            for (int kp = 0; kp < S::BKP; ++kp) mul_pairs<S>(acc, As + kp * S::PA, Bs + kp * S::PB);
        } else {
#pragma unroll 1
            for (int kp = 0; kp < kn; ++kp) mul_pairs<S>(acc, As + kp * S::PA, Bs + kp * S::PB);
        }
        slot = slot + 1 == S::STAGES ? 0 : slot + 1;
        fill = fill + 1 == S::STAGES ? 0 : fill + 1;
    }
#pragma unroll
    for (int i = 0; i < S::TM; ++i) {
        const int m = m0 + mr + kRowThreads * i;
        if (m >= g.Mtot) continue;
        const int l = m / g.Mb, r = m - l * g.Mb;
        float* const C = g.C + (int64_t)l * g.K * g.ldo + r;
        float er = 0.f, lam = 0.f;
        if (PASS == G2_FWD_Y) {
            er = M.ex[r];
            lam = M.lam[l];
        }
#pragma unroll
        for (int j = 0; j < S::TN; ++j) {
            const int n = n0 + nc + S::CT * j;
            if (n >= half) continue;
            const int n2 = g.K - 1 - n;
            float v = acc[i][j].x + acc[i][j].y, w = acc[i][j].x - acc[i][j].y;
            if (PASS == G2_FWD_Y) {
                v = v / (er + M.ey[n] - lam);
                w = w / (er + M.ey[n2] - lam);
            }
            float *pv = C + (int64_t)n * g.ldo, *pw = C + (int64_t)n2 * g.ldo;
            if (PASS == G4_INV_Y && ga.accumulate) {
                v += *pv;
                if (n2 != n) w += *pw;
            }
            *pv = v;
            if (n2 != n) *pw = w;
        }
    }
}

using SimtKernel = void (*)(GemmArgs);
template <class S>
struct Passes {
    static constexpr SimtKernel k[4] = {k_gemm_simt<G1_FWD_X, S>, k_gemm_simt<G2_FWD_Y, S>, k_gemm_simt<G3_INV_X, S>,
                                        k_gemm_simt<G4_INV_Y, S>};
};
struct ShapeInfo {
    int bm, bn, nt;
    size_t smem;
    const SimtKernel* k;
};
template <class S>
constexpr ShapeInfo info() {
    return {S::BM, S::BN, S::NT, S::SMEM, Passes<S>::k};
}
const ShapeInfo kShapes[kSimtShapes] = {info<Shape0>(), info<Shape1>(), info<Shape2>(), info<Shape3>()};
static_assert(Shape0::SMEM <= 48 * 1024 && Shape1::SMEM <= 48 * 1024 && Shape2::SMEM <= 48 * 1024 &&
                  Shape3::SMEM <= 48 * 1024,
              "no opt-in to more shared memory");

}  // namespace

int simt_tile_rows(int shape) { return kShapes[shape].bm; }
int simt_tile_cols(int shape) { return 2 * kShapes[shape].bn; }
int simt_row_tiles(int shape, int rows) { return (rows + kShapes[shape].bm - 1) / kShapes[shape].bm; }
int simt_col_tiles(int shape, int n) { return ((n + 1) / 2 + kShapes[shape].bn - 1) / kShapes[shape].bn; }

// The shape with the least work on the busiest SM: tiles per SM (rounded up) times the tile's
// area, weighted by what a unit of area cost with that shape on members that fill the GPU
// (the small shapes read more shared memory per multiply-add); the smaller shape on a tie, for
// its shorter sums per thread.  Measured per pass on GB300 (the choice, the best other shape and
// the 64 x 64 plain product before this kernel): 3-layer 130^2 8.3 / 8.4 / 18.4 us (16 x 8),
// 3-layer 258^2 11.3 / 12.8 / 29.1 us (32 x 24), 3-layer 514^2 23.4 / 24.8 / 65.7 us (64 x 48),
// 5-layer 502 x 702 44.3 / 50.0 / 108 us (64 x 24), 3-layer 1026^2 102 / 128 / 337 us (64 x 48);
// each figure holds ~5 us of event overhead.
int simt_shape(const int64_t (&tiles)[kSimtShapes], int n_sm) {
    constexpr int weight[kSimtShapes] = {10, 12, 13, 20};
    int best = 0;
    int64_t least = 0;
    for (int k = 0; k < kSimtShapes; ++k) {
        const int64_t cost = (tiles[k] + n_sm - 1) / n_sm * kShapes[k].bm * kShapes[k].bn * weight[k];
        if (k == 0 || cost <= least) {
            best = k;
            least = cost;
        }
    }
    return best;
}

cudaError_t launch_gemm_simt(const GemmArgs& g, int shape, int ntiles, cudaStream_t s, bool pdl) {
    if (shape < 0 || shape >= kSimtShapes || g.pass < G1_FWD_X || g.pass > G4_INV_Y) return cudaErrorInvalidValue;
    const ShapeInfo& i = kShapes[shape];
    return launch_k(i.k[g.pass], ntiles, i.nt, i.smem, s, pdl, g);
}

}  // namespace qg

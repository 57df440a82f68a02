// evaluate.cu -- point evaluation of sparse-grid DG expansions on the GPU.
//
// reconstruct_DG (src/dg_methods.jl:150-165) sums, over every level block L,
// the k^D coefficients of the one cell of L that contains x, times the
// tensor-product basis V = prod_d v(k, L_d - 1, cell_d, m_d, x_d)
// (src/dg_methods.jl:27-35, 45-53) with cell_d = cell_index(x_d, L_d - 1)
// (src/dg_methods.jl:70-78):
//   level 0:  v = sqrt(2) P_{m-1}(2x - 1)
//   level l:  v = sqrt(2^l) h_m(2^l x - (2 cell - 1)),  h the multiwavelet
//             piece for y < 0 or y >= 0, zero for |y| > 1 (array2poly,
//             src/1d_dg_functions.jl:15-27).
// Two kernels.  k_evaluate, one warp per point: the lanes first tabulate the k 1D
// values and the cell of every (dimension, level) in shared memory, then
// split the level blocks among themselves and contract each block's k^D
// coefficients one dimension at a time; a shuffle tree sums the lanes.  For
// k <= 5 and kPencilPoints points or more, k_lines first sums the levels along
// dimension 1 once for all points, and k_evaluate_pencils adds up one block per
// pencil (see there).  All arithmetic is FP64, like the reference.  A coordinate below 0 (or NaN)
// has no cell in the reference (an out-of-range index there) and is reported
// as SGDG_EINVAL; above 1 the last cell is used and |y| > 1 gives zero, as
// in the reference.
#include <cuda_runtime.h>

#include <cmath>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>

#include "api_util.h"
#include "device_util.h"

namespace sgdg {
namespace {

constexpr int kEvalWarps = 4;  // warps (points in flight) per CTA

struct EvalShape {
    int D, k, n, nlev;
    int64_t kD;
    const int8_t* levels;      // nlev x D, 1-based
    const int32_t* lev_off;    // nlev
    const double* pieces;      // 3 k x k: level 0, level >= 1 left (y < 0), right (y >= 0); monomials in y
};

__device__ __forceinline__ double pow2(int j) { return __hiloint2double((1023 + j) << 20, 0); }

__global__ void __launch_bounds__(32 * kEvalWarps)
    k_evaluate(EvalShape S, const double* __restrict__ coeffs, int64_t npts, const double* __restrict__ xs,
               double* __restrict__ out, int* err) {
    extern __shared__ double esm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nl = S.n + 1;  // levels per dimension (0-based level 0..n)
    const int tsz = S.D * nl * S.k;
    double* tab = esm + (size_t)warp * (tsz + S.D * nl);  // [d][l][m] values, then [d][l] cells (0-based)
    double* cel = tab + tsz;
    const int k = S.k;
    for (int64_t p = (int64_t)blockIdx.x * kEvalWarps + warp; p < npts; p += (int64_t)gridDim.x * kEvalWarps) {
        for (int e = lane; e < tsz; e += 32) {
            const int d = e / (nl * k), r = e - d * nl * k, l = r / k, m = r - l * k;
            const double x = xs[p * S.D + d];
            if (!(x >= 0.0)) {  // below 0 or NaN
                atomicExch(err, 1);
                tab[e] = 0.0;
                if (m == 0) cel[d * nl + l] = 0.0;
                continue;
            }
            // cell_index(x, l): 1 for l <= 1; 2^(l-1) for x >= 1; else 1 + floor(2^(l-1) x)
            int cell = 1;
            if (l > 1) cell = x >= 1.0 ? (1 << (l - 1)) : 1 + (int)floor(pow2(l - 1) * x);
            double y, scale;
            const double* pc;
            if (l == 0) {
                y = 2.0 * x - 1.0;
                scale = 1.4142135623730951;  // sqrt(2)
                pc = S.pieces + m * k;
            } else {
                y = pow2(l) * x - (double)(2 * cell - 1);
                scale = (l & 1) ? 1.4142135623730951 * pow2(l >> 1) : pow2(l >> 1);  // sqrt(2^l)
                pc = S.pieces + (y < 0.0 ? 1 : 2) * k * k + m * k;
            }
            double s = 0.0;
            if (fabs(y) <= 1.0)
                for (int i = k - 1; i >= 0; i--) s = s * y + pc[i];
            tab[e] = scale * s;
            if (m == 0) cel[d * nl + l] = (double)(cell - 1);
        }
        __syncwarp();
        double acc = 0.0;
        for (int t = lane; t < S.nlev; t += 32) {
            const int8_t* L = S.levels + (size_t)t * S.D;
            int64_t cl = 0, stride = 1;
            for (int d = 0; d < S.D; d++) {
                cl += (int64_t)cel[d * nl + L[d] - 1] * stride;
                stride <<= (L[d] > 2 ? L[d] - 2 : 0);
            }
            const double* c = coeffs + S.lev_off[t] + S.kD * cl;
            const double* v0 = tab + (L[0] - 1) * k;
            int mo[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            if (S.D >= 3) {
                // outer modes (m_2 .. m_{D-1}, m_2 fastest) times the sum over
                // m_1 of v_1 times the inner sum over m_0: dimensions 0 and 1
                // contracted before the outer product (k^(D-2) (k^2 + k + D - 2)
                // FP64 operations per block instead of k^(D-1) (k + D - 1))
                const double* v1 = tab + (nl + L[1] - 1) * k;
                const int64_t nout = S.kD / (k * k);
                for (int64_t o = 0; o < nout; o++) {
                    double prod = 1.0;
                    for (int d = 2; d < S.D; d++) prod *= tab[(d * nl + L[d] - 1) * k + mo[d]];
                    const double* co = c + o * k * k;
                    double s1 = 0.0;
                    for (int m1 = 0; m1 < k; m1++) {
                        double s0 = 0.0;
                        for (int m0 = 0; m0 < k; m0++) s0 = fma(v0[m0], co[m1 * k + m0], s0);
                        s1 = fma(v1[m1], s0, s1);
                    }
                    acc = fma(prod, s1, acc);
                    for (int d = 2; d < S.D; d++) {  // next outer mode
                        if (++mo[d] < k) break;
                        mo[d] = 0;
                    }
                }
            } else {
                // outer modes (m_1 .. m_{D-1}, m_1 fastest) times the inner sum over m_0
                const int64_t nout = S.kD / k;
                for (int64_t o = 0; o < nout; o++) {
                    double prod = 1.0;
                    for (int d = 1; d < S.D; d++) prod *= tab[(d * nl + L[d] - 1) * k + mo[d]];
                    double s0 = 0.0;
                    for (int m0 = 0; m0 < k; m0++) s0 = fma(v0[m0], c[o * k + m0], s0);
                    acc = fma(prod, s0, acc);
                    for (int d = 1; d < S.D; d++) {  // next outer mode
                        if (++mo[d] < k) break;
                        mo[d] = 0;
                    }
                }
            }
        }
        for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
        if (lane == 0) out[p] = acc;
        __syncwarp();
    }
}

// ---- many points ------------------------------------------------------------
// The hierarchical functions of a line along dimension 1 (levels 1..lmax, equal
// in everything else) are piecewise polynomials on its 2^(lmax-1) finest
// pieces, so the line's k 2^(lmax-1) coefficients can be exchanged for as many
// Legendre coefficients on the pieces (an orthonormal change of basis: Alpert's
// two-scale relations, coarse to fine).  A point then meets one block of k^D
// numbers per pencil -- level tuple of the other dimensions -- instead of one
// per level block: 36 instead of 120 for 3D n=7, and the FP64 operations, which
// bound k_evaluate (61 % of that pipe's peak, 3.50 ms for 2^18 points at k=3),
// fall as much (0.87 ms with that pipe 91 % busy).  A block's numbers are padded to a multiple of 32 bytes and
// loaded 32 bytes at a time: the lanes of a warp are 32 points in blocks of
// their own, so a load costs as many L1 accesses as it has lanes, whatever its
// width.
struct Pencils {
    int D, n, np;
    int inner, pad, outer;   // k^min(D,3), the same rounded up to 4, k^(D-3) (1 for D <= 3)
    const int32_t* lmax;     // per pencil: levels along dimension 1
    const int64_t* base;     // first number of its blocks
    const double* scale;     // product of the scales of its 1D functions (2^(1/2) at level 0 and on the
                             // pieces, 2^(l/2) at l), which k_lines puts into the blocks
    const int8_t* levels;    // D - 1 levels of the other dimensions, 1-based
    const int64_t* item;     // first item (piece, cell and mode of the others) of k_lines; np + 1
    const int32_t* lev_off;  // per pencil n + 1 offsets of its level blocks
    const double* two;       // H_0, H_1, then G_0, G_1 of levels 1..n (k x k each): child b's Legendre
                             // coefficients from the parent's and its wavelets' (two_scale)
    const double* pieces;    // as EvalShape
};

// One item: the k Legendre coefficients of a piece, from the line's root down.
template <int K>
__global__ void __launch_bounds__(256)
    k_lines(Pencils S, const double* __restrict__ c, int64_t kD, double* __restrict__ out, int* nonfinite) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= S.item[S.np]) return;
    int lo = 0, hi = S.np - 1;
    while (lo < hi) {  // last pencil with item <= e
        const int mid = (lo + hi + 1) >> 1;
        if (S.item[mid] <= e) lo = mid; else hi = mid - 1;
    }
    const int lmax = S.lmax[lo];
    const int32_t* off = S.lev_off + (int64_t)lo * (S.n + 1);
    const int64_t km = kD / K;  // modes of the other dimensions, fastest
    const int64_t r = (e - S.item[lo]) / km, mo = (e - S.item[lo]) - r * km;
    const int64_t j = r & ((1ll << (lmax - 1)) - 1), cl = r >> (lmax - 1);  // piece, cells of the others
    double s[K];
#pragma unroll
    for (int m = 0; m < K; m++) s[m] = c[off[0] + kD * cl + K * mo + m];
    bool bad = false;
    for (int t = 1; t < lmax; t++) {
        const int64_t ct = t > 1 ? j >> (lmax - t) : 0;
        const double* d = c + off[t] + kD * (ct + (cl << (t > 1 ? t - 1 : 0))) + K * mo;
        const int b = (j >> (lmax - 1 - t)) & 1;
        const double *H = S.two + b * K * K, *G = S.two + (2 * t + b) * K * K;
        double w[K], x[K];
#pragma unroll
        for (int m = 0; m < K; m++) w[m] = d[m];
#pragma unroll
        for (int i = 0; i < K; i++) {
            double v = 0.0;
#pragma unroll
            for (int m = 0; m < K; m++) v = fma(__ldg(H + i * K + m), s[m], fma(__ldg(G + i * K + m), w[m], v));
            x[i] = v;
        }
#pragma unroll
        for (int i = 0; i < K; i++) s[i] = x[i];
    }
    // within its block: the modes of dimensions 1..3 (padded), then the others
    const int in = S.inner / K;
    double* o = out + S.base[lo] + (int64_t)S.pad * S.outer * (j + (cl << (lmax - 1))) + S.pad * (mo / in) + K * (mo % in);
    const double scale = S.scale[lo];
#pragma unroll
    for (int m = 0; m < K; m++) {
        o[m] = scale * s[m];
        bad = bad || (__double2hiint(s[m]) & 0x7ff00000) == 0x7ff00000;
    }
    if (bad) *nonfinite = 1;
}

constexpr int kPencilPts = 32;    // points of a CTA, one per lane
constexpr int kPencilParts = 4;   // warps that share them, every fourth pencil each

// Values at points: a CTA tabulates the 1D values of its points in shared
// memory ([entry][point]), then each warp adds up its pencils.  Bounds: FP64
// pipe (k^D + k^(D-1) + ... operations per pencil and point, a quarter of it
// the tables), then the gathers.
template <int K, int DI>
__global__ void __launch_bounds__(kPencilPts* kPencilParts)
    k_evaluate_pencils(Pencils S, const double* __restrict__ G, int64_t npts, const double* __restrict__ xs,
                       double* __restrict__ out, int* err) {
    extern __shared__ double esm[];
    constexpr int PT = kPencilPts, PAD = ((DI == 1 ? K : DI == 2 ? K * K : K * K * K) + 3) / 4 * 4;
    const int nl = S.n + 1, D = S.D;
    double* tab = esm;                                              // [(d nl + l) K + m][point]
    double* part = tab + (size_t)D * nl * K * PT;                   // [warp][point]
    int* cell = reinterpret_cast<int*>(part + kPencilParts * PT);   // [d][point]: floor(2^n x)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t p = (int64_t)blockIdx.x * PT + lane;
    for (int e = warp; e < D * nl; e += kPencilParts) {
        const int d = e / nl, l = e - d * nl;  // l: 0-based level; dimension 1: pieces of 2^-l
        const double x = p < npts ? xs[p * D + d] : 0.0;
        double v[K];
#pragma unroll
        for (int m = 0; m < K; m++) v[m] = 0.0;
        if (!(x >= 0.0)) {
            atomicExch(err, 1);
        } else {
            const int cells = d == 0 ? l : l > 1 ? l - 1 : 0;  // log2
            int c = 0;  // 0-based
            if (cells > 0) c = x >= 1.0 ? (1 << cells) - 1 : (int)floor(pow2(cells) * x);
            double y;
            const double* pc;
            if (d == 0 || l == 0) {
                y = pow2(cells + 1) * x - (double)(2 * c + 1);
                pc = S.pieces;
            } else {
                y = pow2(l) * x - (double)(2 * c + 1);
                pc = S.pieces + (y < 0.0 ? 1 : 2) * K * K;
            }
            if (fabs(y) <= 1.0)
#pragma unroll
                for (int m = 0; m < K; m++) {
                    double s = __ldg(pc + m * K + K - 1);
#pragma unroll
                    for (int i = K - 2; i >= 0; i--) s = fma(s, y, __ldg(pc + m * K + i));
                    v[m] = s;
                }
        }
#pragma unroll
        for (int m = 0; m < K; m++) tab[(e * K + m) * PT + lane] = v[m];
        if (l == 0) cell[d * PT + lane] = !(x < 1.0) ? (1 << S.n) - 1 : x > 0.0 ? (int)floor(pow2(S.n) * x) : 0;
    }
    __syncthreads();
    double acc = 0.0;
    for (int q = warp; q < S.np; q += kPencilParts) {
        const int lm = S.lmax[q];
        const int8_t* L = S.levels + q * (D - 1);
        int64_t cl = 0;
        int sh = lm - 1;
        for (int d = 1; d < D; d++) {
            const int lc = L[d - 1] > 2 ? L[d - 1] - 2 : 0;
            cl += (int64_t)(cell[d * PT + lane] >> (S.n - lc)) << sh;
            sh += lc;
        }
        const double* g = G + S.base[q] + (int64_t)PAD * S.outer * ((cell[lane] >> (S.n - (lm - 1))) + cl);
        double v0[K], v1[K], v2[K];
#pragma unroll
        for (int m = 0; m < K; m++) {
            v0[m] = tab[((lm - 1) * K + m) * PT + lane];
            if (DI > 1) v1[m] = tab[((nl + L[0] - 1) * K + m) * PT + lane];
            if (DI > 2) v2[m] = tab[((2 * nl + L[1] - 1) * K + m) * PT + lane];
        }
        for (int o = 0; o < S.outer; o++) {
            double s0 = 0.0, s1 = 0.0, s2 = 0.0;
#pragma unroll
            for (int u = 0; u < PAD; u += 4) {
                double t[4];
                asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
                    : "=d"(t[0]), "=d"(t[1]), "=d"(t[2]), "=d"(t[3]) : "l"(g + (int64_t)o * PAD + u));
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int at = u + i, m0 = at % K, m1 = at / K % K, m2 = at / (K * K);
                    if (at >= (DI == 1 ? K : DI == 2 ? K * K : K * K * K)) continue;
                    s0 = m0 ? fma(v0[m0], t[i], s0) : v0[0] * t[i];
                    if (DI > 1 && m0 == K - 1) {
                        s1 = m1 ? fma(v1[m1], s0, s1) : v1[0] * s0;
                        if (DI > 2 && m1 == K - 1) s2 = m2 ? fma(v2[m2], s1, s2) : v2[0] * s1;
                    }
                }
            }
            double r = DI == 1 ? s0 : DI == 2 ? s1 : s2;
            if (S.outer > 1) {
                int mo = o;
                for (int d = 3; d < D; d++, mo /= K) r *= tab[((d * nl + L[d - 1] - 1) * K + mo % K) * PT + lane];
            }
            acc += r;
        }
    }
    part[warp * PT + lane] = acc;
    __syncthreads();
    if (warp == 0 && p < npts) {
        double s = 0.0;
        for (int w = 0; w < kPencilParts; w++) s += part[w * PT + lane];
        out[p] = s;
    }
}

// Sum over terms of separable products (tensor_construct,
// src/tensor_construct.jl:19-62, and sums of Fourier modes): coefficient i
// of the D-dim vector is  sum_t amp_t * part_t( e^{i phi_t} prod_d Z_td[i_d] )
// with i_d the 1D index of i along d (get_index_1D,
// src/additional_tools.jl:8-13: k * (block of (level, cell)) + mode) and
// part_t the real or imaginary part.  The complex products round each
// product and sum separately, as numpy does.  One thread per coefficient.
struct TermShape {
    int D, k, nlev, nterms;
    int64_t kD, N1, N;
    const int8_t* levels;
    const int32_t* lev_off;
    const double* Z;      // nterms x D x N1 (re, im)
    const double* coef;   // nterms x 4: amp, cos phi, sin phi, part (0 real, 1 imaginary)
};

__global__ void k_tensor_sum(TermShape S, double* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.N) return;
    int lo = 0, hi = S.nlev - 1;
    while (lo < hi) {  // level block holding i
        const int mid = (lo + hi + 1) >> 1;
        if (S.lev_off[mid] <= i) lo = mid; else hi = mid - 1;
    }
    const int8_t* L = S.levels + (size_t)lo * S.D;
    const int64_t local = i - S.lev_off[lo];
    int64_t cl = local / S.kD, ml = local - cl * S.kD;
    int64_t i1[8];
    for (int d = 0; d < S.D; d++) {
        const int64_t nc = (int64_t)1 << (L[d] > 2 ? L[d] - 2 : 0);
        const int64_t c = cl % nc, m = ml % S.k;
        cl /= nc;
        ml /= S.k;
        i1[d] = S.k * ((L[d] >= 2 ? ((int64_t)1 << (L[d] - 2)) : 0) + c) + m;
    }
    double acc = 0.0;
    for (int t = 0; t < S.nterms; t++) {
        const double* cf = S.coef + 4 * t;
        double zr = cf[1], zi = cf[2];
        for (int d = 0; d < S.D; d++) {
            const double* z = S.Z + (((size_t)t * S.D + d) * S.N1 + i1[d]) * 2;
            const double ar = __dsub_rn(__dmul_rn(zr, z[0]), __dmul_rn(zi, z[1]));
            const double ai = __dadd_rn(__dmul_rn(zr, z[1]), __dmul_rn(zi, z[0]));
            zr = ar;
            zi = ai;
        }
        acc = __dadd_rn(acc, __dmul_rn(cf[0], cf[3] != 0.0 ? zi : zr));
    }
    out[i] = acc;
}

// device tables of one (D, k, n, scheme)
struct EvalTables {
    SparseIndex ix;
    DevBuf levels, lev_off, pieces;
    size_t smem = 0;
    // the pencils along dimension 1 (k <= 5), built with the first call that uses them
    std::mutex mu;
    DevBuf lmax, base, scale, plevels, item, plev_off, two;
    Pencils P{};
    int64_t items = 0, numbers = 0;  // of k_lines; of its output
    size_t psmem = 0;
    int refused = -1;  // the budget (g_budget_set) that had no room for them
};

constexpr int kPencilMaxK = 5;
// From these counts of points and of products with a coefficient on, the pencils
// pay for k_lines (us per call, blocks and pencils: 3D k=3 n=7 64 and 69 at 1000
// points, 90 and 69 at 4000, 3495 and 947 at 2^18; 4D k=3 n=4 90 and 104, 138 and
// 105, 6579 and 2190; 2D k=2 n=6 39 and 41 at 4000, 64 and 46 at 16000, 524 and
// 165; 1D k=3 n=8 39 and 45, 55 and 54, 448 and 141.  With the scales in the
// blocks the pencils take 866, 2126, 124 and 100 at 2^18 points).
constexpr int64_t kPencilPoints = 4096, kPencilTerms = 1 << 20;

// H_b[i][m] = int leg_i(z) p_m((z + s) / 2) dz over [-1, 1], s = 2b - 1, p_m the
// parent's Legendre function m, and G_b of level t 2^((t - 1) / 2) times the same of
// the wavelets' polynomials on that half: child b's coefficients without the factor
// 2^(-1/2) of every level, which is 2^(t/2) times what they stand for.  A line goes
// through up to n of the H_b; so their diagonal is 1, 1/2, 1/4..., exactly, and
// the rest is computed in long double and rounded once.  Relative L2 error of the
// values against long double (blocks; pencils in double with the factors; like
// this): 1D k=3 n=10 8.1e-16, 1.8e-15, 7.5e-16; 2D k=2 n=8 3.2e-16, 1.0e-15,
// 3.3e-16; 2D k=4 n=6 1.4e-15, 2.0e-15, 1.1e-15; 3D k=3 n=7 1.15e-15, 1.31e-15,
// 1.14e-15.  The wavelets are the blocks', rounded as they are.
std::vector<double> two_scale(int k, int n) {
    using Real = long double;
    using Poly = std::vector<Real>;  // monomials in [-1, 1]
    std::vector<Poly> leg(k, Poly(k, 0));
    for (int m = 0; m < k; m++) {
        if (m < 2) leg[m][m] = 1;
        for (int i = 0; m >= 2 && i < k; i++)
            leg[m][i] = ((2 * m - 1) * (i > 0 ? leg[m - 1][i - 1] : 0) - (m - 1) * leg[m - 2][i]) / m;
    }
    for (int m = 0; m < k; m++)
        for (Real& c : leg[m]) c *= std::sqrt(Real(2 * m + 1) / 2);
    std::vector<double> out((size_t)2 * (n + 1) * k * k);
    for (int b = 0; b < 2; b++)
        for (int g = 0; g < 2; g++)
            for (int m = 0; m < k; m++) {
                const HierFn f = make_hier_fn(k, 1, 1, m + 1);
                const Poly wav(b ? f.right : f.left, (b ? f.right : f.left) + k);
                const Poly& p = g ? wav : leg[m];
                Poly q(k, 0);  // p((z + s) / 2) in z, by Horner
                for (int i = k - 1; i >= 0; i--) {
                    Poly t(k, 0);
                    for (int a = 0; a < k; a++) {
                        t[a] += Real(2 * b - 1) / 2 * q[a];
                        if (a + 1 < k) t[a + 1] += q[a] / 2;
                    }
                    t[0] += p[i];
                    q = t;
                }
                for (int i = 0; i < k; i++) {
                    Real v = 0;
                    for (int a = 0; a < k; a++)
                        for (int c = 0; c < k; c++)
                            if ((a + c) % 2 == 0) v += leg[i][a] * q[c] * 2 / (a + c + 1);
                    if (g == 0) out[(size_t)b * k * k + i * k + m] = (double)v;
                    for (int t = 1; g == 1 && t <= n; t++)
                        out[(size_t)(2 * t + b) * k * k + i * k + m] = (double)(std::sqrt(std::ldexp(Real(1), t - 1)) * v);
                }
            }
    return out;
}

void build_pencils(EvalTables& T) {
    const SparseIndex& ix = T.ix;
    const int D = ix.D, k = ix.k, n = ix.n;
    Pencils P{};
    P.D = D;
    P.n = n;
    P.inner = 1;
    P.outer = 1;
    for (int d = 0; d < D; d++) (d < 3 ? P.inner : P.outer) *= k;
    P.pad = (P.inner + 3) / 4 * 4;
    std::vector<int32_t> lmax, off;
    std::vector<int64_t> base, item(1, 0);
    std::vector<int8_t> lev;
    std::vector<double> scale;
    int64_t numbers = 0;
    int L[kDMax];
    for (int b = 0; b < ix.nlev; b++) {
        const int* Lb = &ix.levels[(size_t)b * D];
        if (Lb[0] != 1) continue;
        for (int d = 0; d < D; d++) L[d] = Lb[d];
        int lm = 0;
        for (int l = 1; l <= n + 1; l++) {
            L[0] = l;
            if (ix.cut(L)) {
                off.push_back(0);
                continue;
            }
            off.push_back((int32_t)ix.lev_off[ix.lookup_level(L)]);
            lm = l;
        }
        int half = 1;  // log2 of the square of the scale
        for (int d = 1; d < D; d++) {
            lev.push_back((int8_t)Lb[d]);
            half += std::max(1, Lb[d] - 1);
        }
        scale.push_back(std::ldexp(half % 2 ? std::sqrt(2.0) : 1.0, half / 2));
        lmax.push_back(lm);
        base.push_back(numbers);
        const int64_t blocks = ix.lev_cells[b] << (lm - 1);  // finest pieces x cells of the others
        numbers += blocks * P.pad * P.outer;
        item.push_back(item.back() + blocks * (ix.kD / k));
    }
    T.lmax = upload(lmax, nullptr);
    T.base = upload(base, nullptr);
    T.scale = upload(scale, nullptr);
    T.plevels = upload(lev, nullptr);
    T.item = upload(item, nullptr);
    T.plev_off = upload(off, nullptr);
    T.two = upload(two_scale(k, n), nullptr);
    CK(cudaStreamSynchronize(nullptr));
    P.lmax = T.lmax.as<int32_t>();
    P.base = T.base.as<int64_t>();
    P.scale = T.scale.as<double>();
    P.levels = T.plevels.as<int8_t>();
    P.item = T.item.as<int64_t>();
    P.lev_off = T.plev_off.as<int32_t>();
    P.two = T.two.as<double>();
    P.pieces = T.pieces.as<double>();
    T.items = item.back();
    T.numbers = numbers;
    T.psmem = sizeof(double) * kPencilPts * ((size_t)D * (n + 1) * k + kPencilParts) + sizeof(int) * kPencilPts * D;
    P.np = (int)lmax.size();
    T.P = P;
}

// null where there is no room for them, now or earlier under the same budget
const Pencils* eval_pencils(EvalTables& T) {
    std::lock_guard<std::mutex> g(T.mu);
    if (T.P.np > 0) return &T.P;
    if (T.refused == g_budget_set.load()) return nullptr;
    try {
        build_pencils(T);
        return &T.P;
    } catch (const Error& e) {
        if (e.code != SGDG_ENOMEM_BUDGET) throw;
    }
    for (DevBuf* b : {&T.lmax, &T.base, &T.scale, &T.plevels, &T.item, &T.plev_off, &T.two}) b->release();
    T.refused = g_budget_set.load();
    return nullptr;
}

template <int K>
cudaError_t launch_pencils(const EvalTables& T, const Pencils& P, const double* coeffs, int64_t npts, const double* xs,
                           double* out, double* G, int* err, cudaStream_t st) {
    k_lines<K><<<(unsigned)((T.items + 255) / 256), 256, 0, st>>>(P, coeffs, T.ix.kD, G, err + 1);
    auto kernel = P.D == 1 ? k_evaluate_pencils<K, 1> : P.D == 2 ? k_evaluate_pencils<K, 2> : k_evaluate_pencils<K, 3>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    kernel<<<(unsigned)((npts + kPencilPts - 1) / kPencilPts), kPencilPts * kPencilParts, T.psmem, st>>>(P, G, npts, xs, out,
                                                                                                      err);
    return cudaGetLastError();
}

std::mutex g_eval_mu;
std::map<std::tuple<int, int, int, int>, std::unique_ptr<EvalTables>> g_eval;

EvalTables& eval_tables(int D, int k, int n, int scheme) {
    std::lock_guard<std::mutex> g(g_eval_mu);
    auto key = std::make_tuple(D, k, n, scheme);
    auto f = g_eval.find(key);
    if (f != g_eval.end()) return *f->second;
    std::unique_ptr<EvalTables> T(new EvalTables);
    T->ix = make_index(D, k, n, scheme);
    const SparseIndex& ix = T->ix;
    std::vector<int8_t> lv(ix.levels.size());
    for (size_t i = 0; i < lv.size(); i++) lv[i] = (int8_t)ix.levels[i];
    std::vector<int32_t> lo(ix.lev_off.begin(), ix.lev_off.end());
    std::vector<double> pc((size_t)3 * k * k, 0.0);
    for (int m = 1; m <= k; m++) {
        const HierFn f0 = make_hier_fn(k, 0, 1, m), f1 = make_hier_fn(k, 1, 1, m);
        for (int i = 0; i < k; i++) {
            pc[(size_t)(m - 1) * k + i] = f0.left[i];
            pc[(size_t)k * k + (m - 1) * k + i] = f1.left[i];
            pc[(size_t)2 * k * k + (m - 1) * k + i] = f1.right[i];
        }
    }
    T->levels = upload(lv, nullptr);
    T->lev_off = upload(lo, nullptr);
    T->pieces = upload(pc, nullptr);
    CK(cudaStreamSynchronize(nullptr));
    T->smem = sizeof(double) * (size_t)kEvalWarps * ((size_t)D * (n + 1) * k + (size_t)D * (n + 1));
    EvalTables& r = *T;
    g_eval.emplace(key, std::move(T));
    return r;
}

void evaluate_impl(int D, int k, int n, int scheme, const double* coeffs, int64_t npts, const double* xs,
                   double* out, cudaStream_t st) {
    if (npts < 0) throw Error(SGDG_EINVAL, "npts must be >= 0");
    EvalTables& T = eval_tables(D, k, n, scheme);
    if (npts == 0) return;
    if (k <= kPencilMaxK && npts >= kPencilPoints && npts * T.ix.nlev * T.ix.kD >= kPencilTerms &&
        npts < (int64_t(1) << 31) * kPencilPts) {
        const Pencils* P = eval_pencils(T);
        DevBuf work;
        if (P && T.psmem <= 200 * 1024) try {
                work.alloc(sizeof(double) * (size_t)T.numbers + 2 * sizeof(int));
            } catch (const Error&) {  // no room: k_evaluate needs none
            }
        if (work.p) {
            int* err = reinterpret_cast<int*>(work.as<double>() + T.numbers);
            CK(cudaMemsetAsync(err, 0, 2 * sizeof(int), st));
            auto launch = k == 1 ? launch_pencils<1> : k == 2 ? launch_pencils<2> : k == 3 ? launch_pencils<3>
                        : k == 4 ? launch_pencils<4> : launch_pencils<5>;
            CK(launch(T, *P, coeffs, npts, xs, out, work.as<double>(), err, st));
            int h[2] = {0, 0};
            CK(cudaMemcpyAsync(h, err, sizeof(h), cudaMemcpyDeviceToHost, st));
            CK(cudaStreamSynchronize(st));
            work.recycle();
            if (h[0]) throw Error(SGDG_EINVAL, "a point coordinate is below 0 or NaN (no cell contains it)");
            if (!h[1]) return;
            // a coefficient that is not finite: block by block, as the sum over levels spreads it
        }
    }
    if (T.smem > 200 * 1024) throw Error(SGDG_EUNSUPPORTED, "point tables exceed shared memory");
    static bool configured = false;
    if (!configured) {
        CK(cudaFuncSetAttribute(k_evaluate, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        configured = true;
    }
    EvalShape S{D, k, n, T.ix.nlev, T.ix.kD, T.levels.as<int8_t>(), T.lev_off.as<int32_t>(), T.pieces.as<double>()};
    DevBuf err(sizeof(int));
    CK(cudaMemsetAsync(err.p, 0, sizeof(int), st));
    int dev = 0, sms = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int64_t need = (npts + kEvalWarps - 1) / kEvalWarps;
    const int grid = (int)std::min<int64_t>(need, (int64_t)sms * 16);
    k_evaluate<<<grid, 32 * kEvalWarps, T.smem, st>>>(S, coeffs, npts, xs, out, err.as<int>());
    CK(cudaGetLastError());
    int h_err = 0;
    CK(cudaMemcpyAsync(&h_err, err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    err.recycle();
    if (h_err) throw Error(SGDG_EINVAL, "a point coordinate is below 0 or NaN (no cell contains it)");
}

void tensor_sum_impl(int D, int k, int n, int scheme, int nterms, const double* Z, const double* coef, double* out,
                     cudaStream_t st) {
    const EvalTables& T = eval_tables(D, k, n, scheme);
    TermShape S{D, k, T.ix.nlev, nterms, T.ix.kD, (int64_t)k << n, T.ix.N, T.levels.as<int8_t>(),
                T.lev_off.as<int32_t>(), Z, coef};
    k_tensor_sum<<<(int)((T.ix.N + 255) / 256), 256, 0, st>>>(S, out);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(st));
}

void check_shape(int D, int k, int n) {
    if (D < 1 || D > 8) throw Error(SGDG_EINVAL, "D must be in 1..8");
    if (k < 1 || k > kKMax) throw Error(SGDG_EINVAL, "k must be in 1..10");
    if (n < 0 || n > 24) throw Error(SGDG_EINVAL, "n must be in 0..24");
}

}  // namespace
}  // namespace sgdg

using namespace sgdg;

extern "C" {

int sgdg_evaluate(int D, int k, int n, int scheme, const double* coeffs, int64_t npts, const double* xs,
                  double* values) {
    API_BEGIN
    check_shape(D, k, n);
    NEED(coeffs);
    if (npts > 0) {
        NEED(xs);
        NEED(values);
    }
    require_gpu();
    const SparseIndex& ix = eval_tables(D, k, n, scheme).ix;
    if (npts == 0) return SGDG_OK;
    cudaStream_t st = nullptr;
    DevBuf dc(sizeof(double) * ix.N), dx(sizeof(double) * (size_t)npts * D), dv(sizeof(double) * (size_t)npts);
    CK(cudaMemcpyAsync(dc.p, coeffs, sizeof(double) * ix.N, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(dx.p, xs, sizeof(double) * (size_t)npts * D, cudaMemcpyHostToDevice, st));
    evaluate_impl(D, k, n, scheme, dc.as<double>(), npts, dx.as<double>(), dv.as<double>(), st);
    CK(cudaMemcpyAsync(values, dv.p, sizeof(double) * (size_t)npts, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    for (DevBuf* b : {&dc, &dx, &dv}) b->recycle();
    API_END
}

int sgdg_tensor_sum(int D, int k, int n, int scheme, int nterms, const double* Z, const double* coef, double* out) {
    API_BEGIN
    check_shape(D, k, n);
    if (nterms < 1) throw Error(SGDG_EINVAL, "nterms must be >= 1");
    NEED(Z);
    NEED(coef);
    NEED(out);
    require_gpu();
    const SparseIndex& ix = eval_tables(D, k, n, scheme).ix;
    const size_t zlen = (size_t)nterms * D * ((size_t)k << n) * 2;
    cudaStream_t st = nullptr;
    DevBuf dz(sizeof(double) * zlen), dc(sizeof(double) * 4 * (size_t)nterms), dout(sizeof(double) * ix.N);
    CK(cudaMemcpyAsync(dz.p, Z, sizeof(double) * zlen, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(dc.p, coef, sizeof(double) * 4 * nterms, cudaMemcpyHostToDevice, st));
    tensor_sum_impl(D, k, n, scheme, nterms, dz.as<double>(), dc.as<double>(), dout.as<double>(), st);
    CK(cudaMemcpyAsync(out, dout.p, sizeof(double) * ix.N, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    API_END
}

int sgdg_evaluate_device(int D, int k, int n, int scheme, const double* coeffs_dev, int64_t npts,
                         const double* xs_dev, double* values_dev, void* stream) {
    API_BEGIN
    check_shape(D, k, n);
    NEED(coeffs_dev);
    if (npts > 0) {
        NEED(xs_dev);
        NEED(values_dev);
    }
    require_gpu();
    evaluate_impl(D, k, n, scheme, coeffs_dev, npts, xs_dev, values_dev, (cudaStream_t)stream);
    API_END
}

}  // extern "C"

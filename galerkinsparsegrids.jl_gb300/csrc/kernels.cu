// kernels.cu -- the plain form and small helpers.
//
//  * k_csr: FP64 CSR mat-vec (the closure body *(RHS, x) of src/pdes.jl:63)
//    over NV vectors in one pass over A (the passes fused with the RK4 stage
//    update are in csr_step.cu).  Rows are binned by length
//    (DevCSR.bin_*): a row of bin b gets 2^b lanes with at most eight entries
//    each (four in flight), so the short and the long rows of one matrix (the
//    nodal transforms hold both) keep the lanes equally busy and the lane
//    reduction (csr_reduce) stays small against the FMAs -- on GB300 both run
//    on the FP64 pipe, which bounds these kernels; every block of the grid
//    serves one bin.  Rows longer than A.split are summed by
//    k_csr_segments (one warp per segment) and k_csr_long_rows (segment
//    partials in order, then the same epilogue).
//    Element (j, i) of the vector set x is x[i * xi + j * xs]: xi = 1 and
//    xs = length for vectors one after another, xi = count and xs = 1 for
//    interleaved vectors, whose values at one column share a sector and come
//    in as one 32-byte (W = 4) or 16-byte (W = 2) load.
//  * k_vlasov_points: the point-basis combination of the Vlasov right-hand side.
//  * k_f64_to_f32 / k_f32_to_f64: precision conversions of whole vectors.
#include <cuda_runtime.h>

#include <cstdint>

#include "bounds.cuh"
#include "csr.cuh"
#include "engine.h"

namespace sgdg {

// 256-bit read-only load (sm_100 and later); p 32-byte aligned
__device__ __forceinline__ void ld_nc_v4(const double* p, double& a, double& b, double& c, double& d) {
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a), "=d"(b), "=d"(c), "=d"(d) : "l"(p));
}

// the values of NV vectors at one column (element offset off = column * xi),
// W adjacent vectors per load (W = 2: 16-byte, W = 4: 32-byte aligned)
template <int NV, int W>
__device__ __forceinline__ void csr_gather(const double* __restrict__ x, int64_t off, int64_t xs, double (&v)[NV]) {
    if constexpr (W == 4) {
#pragma unroll
        for (int j = 0; j < NV; j += 4) ld_nc_v4(x + off + j, v[j], v[j + 1], v[j + 2], v[j + 3]);
    } else if constexpr (W == 2) {
#pragma unroll
        for (int j = 0; j < NV; j += 2) {
            const double2 t = __ldg(reinterpret_cast<const double2*>(x + off + j));
            v[j] = t.x;
            v[j + 1] = t.y;
        }
    } else {
#pragma unroll
        for (int j = 0; j < NV; j++) v[j] = __ldg(x + off + j * xs);
    }
}

// s[j] = row `row` of A times vector j, summed over VS lanes (row < 0: zeros,
// but the lanes still take part in the shuffles); see csr_reduce for where
// the sums end up
template <int VS, int NV, int W>
__device__ __forceinline__ void csr_row(const DevCSR& A, int64_t row, const double* __restrict__ x, int64_t xi,
                                        int64_t xs, int lane, double (&s)[NV]) {
#pragma unroll
    for (int j = 0; j < NV; j++) s[j] = 0.0;
    if (row >= 0) {
        const int64_t b = A.rowptr[row], e = A.rowptr[row + 1];
        int64_t p = b + lane;
        // four entries per lane in flight: the column loads, then the gathers of x
        for (; p + 3 * VS < e; p += 4 * VS) {
            int c0 = __ldg(A.col + p), c1 = __ldg(A.col + p + VS), c2 = __ldg(A.col + p + 2 * VS),
                c3 = __ldg(A.col + p + 3 * VS);
            if (!SGDG_IN(c0, A.m)) c0 = 0;  // debug build: counted, read column 0 instead
            if (!SGDG_IN(c1, A.m)) c1 = 0;
            if (!SGDG_IN(c2, A.m)) c2 = 0;
            if (!SGDG_IN(c3, A.m)) c3 = 0;
            const double v0 = __ldg(A.val + p), v1 = __ldg(A.val + p + VS), v2 = __ldg(A.val + p + 2 * VS),
                         v3 = __ldg(A.val + p + 3 * VS);
            double x0[NV], x1[NV], x2[NV], x3[NV];
            csr_gather<NV, W>(x, c0 * xi, xs, x0);
            csr_gather<NV, W>(x, c1 * xi, xs, x1);
            csr_gather<NV, W>(x, c2 * xi, xs, x2);
            csr_gather<NV, W>(x, c3 * xi, xs, x3);
#pragma unroll
            for (int j = 0; j < NV; j++) {
                s[j] = fma(v0, x0[j], s[j]);
                s[j] = fma(v1, x1[j], s[j]);
                s[j] = fma(v2, x2[j], s[j]);
                s[j] = fma(v3, x3[j], s[j]);
            }
        }
        for (; p < e; p += VS) {
            int c = __ldg(A.col + p);
            if (!SGDG_IN(c, A.m)) c = 0;
            const double v = __ldg(A.val + p);
            double xv[NV];
            csr_gather<NV, W>(x, c * xi, xs, xv);
#pragma unroll
            for (int j = 0; j < NV; j++) s[j] = fma(v, xv[j], s[j]);
        }
    }
    csr_reduce<VS, NV>(s, lane);
}

// the rows of bin `bin`, 2^bin = VS lanes each
template <int VS, int NV, int W>
__device__ __forceinline__ void csr_bin(const DevCSR& A, int bin, int64_t rb, const double* __restrict__ x, int64_t xi,
                                        int64_t xs, double* y, int64_t yi, int64_t ys) {
    const int64_t t = (rb - A.bin_block[bin]) * blockDim.x + threadIdx.x;
    const int64_t idx = t / VS, first = A.bin_first[bin];
    const int lane = int(t % VS);
    int64_t row = idx < A.bin_first[bin + 1] - first ? (int64_t)A.bin_rows[first + idx] : -1;
    if (row >= 0 && !SGDG_IN(row, A.m)) row = -1;
    double s[NV];
    csr_row<VS, NV, W>(A, row, x, xi, xs, lane, s);
    bool stores;
    const int owner = csr_owner<VS, NV>(lane, stores);
    if (row >= 0 && stores) {
        if (owner >= 0)
            y[row * yi + owner * ys] = s[0];
        else {
#pragma unroll
            for (int j = 0; j < NV; j++) y[row * yi + j * ys] = s[j];
        }
    }
}

template <int NV, int W>
__global__ void __launch_bounds__(256) k_csr(DevCSR A, const double* __restrict__ x, int64_t xi, int64_t xs,
                                             double* y, int64_t yi, int64_t ys) {
    const int64_t rb = blockIdx.x;
    int bin = 0;
    while (bin + 1 < kCsrBins && rb >= A.bin_block[bin + 1]) bin++;
    switch (bin) {
        case 0: csr_bin<1, NV, W>(A, 0, rb, x, xi, xs, y, yi, ys); break;
        case 1: csr_bin<2, NV, W>(A, 1, rb, x, xi, xs, y, yi, ys); break;
        case 2: csr_bin<4, NV, W>(A, 2, rb, x, xi, xs, y, yi, ys); break;
        case 3: csr_bin<8, NV, W>(A, 3, rb, x, xi, xs, y, yi, ys); break;
        case 4: csr_bin<16, NV, W>(A, 4, rb, x, xi, xs, y, yi, ys); break;
        default: csr_bin<32, NV, W>(A, 5, rb, x, xi, xs, y, yi, ys); break;
    }
}

// one warp per segment of a long row; partial sums of vector j at
// A.partial[j * A.nseg + seg]
template <int NV, int W>
__global__ void __launch_bounds__(256) k_csr_segments(DevCSR A, const double* __restrict__ x, int64_t xi,
                                                      int64_t xs) {
    const int64_t seg = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (seg >= A.nseg) return;
    double s[NV];
#pragma unroll
    for (int j = 0; j < NV; j++) s[j] = 0.0;
    const int64_t e = A.seg_end[seg];
    int64_t p = A.seg_begin[seg] + lane;
    for (; p + 96 < e; p += 128) {
        int c0 = __ldg(A.col + p), c1 = __ldg(A.col + p + 32), c2 = __ldg(A.col + p + 64), c3 = __ldg(A.col + p + 96);
        if (!SGDG_IN(c0, A.m)) c0 = 0;
        if (!SGDG_IN(c1, A.m)) c1 = 0;
        if (!SGDG_IN(c2, A.m)) c2 = 0;
        if (!SGDG_IN(c3, A.m)) c3 = 0;
        const double v0 = __ldg(A.val + p), v1 = __ldg(A.val + p + 32), v2 = __ldg(A.val + p + 64),
                     v3 = __ldg(A.val + p + 96);
        double x0[NV], x1[NV], x2[NV], x3[NV];
        csr_gather<NV, W>(x, c0 * xi, xs, x0);
        csr_gather<NV, W>(x, c1 * xi, xs, x1);
        csr_gather<NV, W>(x, c2 * xi, xs, x2);
        csr_gather<NV, W>(x, c3 * xi, xs, x3);
#pragma unroll
        for (int j = 0; j < NV; j++) {
            s[j] = fma(v0, x0[j], s[j]);
            s[j] = fma(v1, x1[j], s[j]);
            s[j] = fma(v2, x2[j], s[j]);
            s[j] = fma(v3, x3[j], s[j]);
        }
    }
    for (; p < e; p += 32) {
        int c = __ldg(A.col + p);
        if (!SGDG_IN(c, A.m)) c = 0;
        const double v = __ldg(A.val + p);
        double xv[NV];
        csr_gather<NV, W>(x, c * xi, xs, xv);
#pragma unroll
        for (int j = 0; j < NV; j++) s[j] = fma(v, xv[j], s[j]);
    }
    csr_reduce<32, NV>(s, lane);
    bool stores;
    const int owner = csr_owner<32, NV>(lane, stores);
    if (stores) {
        if (owner >= 0)
            A.partial[owner * A.nseg + seg] = s[0];
        else {
#pragma unroll
            for (int j = 0; j < NV; j++) A.partial[j * A.nseg + seg] = s[j];
        }
    }
}

// one thread per (long row, vector): the row's segment partials in order
__global__ void k_csr_long_rows(DevCSR A, int nv, double* y, int64_t yi, int64_t ys) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= A.nlong * nv) return;
    const int64_t i = t % A.nlong;
    const int j = int(t / A.nlong);
    double s = 0.0;
    for (int q = A.long_seg[i]; q < A.long_seg[i + 1]; q++) s += A.partial[j * A.nseg + q];
    const int64_t row = A.long_row[i];
    if (!SGDG_IN(row, A.m)) return;
    y[row * yi + j * ys] = s;
}

__global__ void k_f64_to_f32(const double* __restrict__ a, float* __restrict__ b, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}

__global__ void k_f32_to_f64(const float* __restrict__ a, double* __restrict__ b, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = (double)a[i];
}

// Vlasov right-hand side in the point basis (src/pdes.jl:185-191): with the
// 2D transformed derivatives interleaved, pt[i * 2D + d] (x dimensions d < D,
// then p),
//   out = -(sum_d v_d .* pt_d) + sum_d F_d .* pt_{D+d},
// each sum left to right with separate roundings of products and sums.
__global__ void k_vlasov_points(const double* __restrict__ v, const double* __restrict__ F,
                                const double* __restrict__ pt, int D, int64_t n, double* __restrict__ out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double* q = pt + i * 2 * D;
        double c1 = __dmul_rn(v[i], q[0]), c2 = __dmul_rn(F[i], q[D]);
        for (int d = 1; d < D; d++) {
            c1 = __dadd_rn(c1, __dmul_rn(v[d * n + i], q[d]));
            c2 = __dadd_rn(c2, __dmul_rn(F[d * n + i], q[D + d]));
        }
        out[i] = __dadd_rn(-c1, c2);
    }
}

SGDG_BOUNDS_READER(csr_bounds_violations)

// ------------------------------------------------------------ launchers ----
static int grid_for(int64_t threads) {
    int64_t b = (threads + 255) / 256;
    return (int)(b > (1LL << 30) ? (1LL << 30) : (b < 1 ? 1 : b));
}

template <int NV, int W>
static void csr_pass(const DevCSR& A, const double* x, int64_t xi, int64_t xs, double* y, int64_t yi, int64_t ys,
                     cudaStream_t st) {
    if (A.bin_block[kCsrBins] > 0)
        k_csr<NV, W><<<A.bin_block[kCsrBins], 256, 0, st>>>(A, x, xi, xs, y, yi, ys);
    if (A.nlong > 0) {
        k_csr_segments<NV, W><<<grid_for(A.nseg * 32), 256, 0, st>>>(A, x, xi, xs);
        k_csr_long_rows<<<grid_for(A.nlong * NV), 256, 0, st>>>(A, NV, y, yi, ys);
    }
}

cudaError_t launch_csr_spmv(const DevCSR& A, const double* x, double* y, cudaStream_t st) {
    csr_pass<1, 1>(A, x, 1, 0, y, 1, 0, st);
    return cudaGetLastError();
}

// y_j = A x_j for j < nv, kCsrMaxVec vectors per pass over A; element (j, i)
// of x at x[i * xi + j * xs], of y at y[i * yi + j * ys]
cudaError_t launch_csr_spmv_multi(const DevCSR& A, int nv, const double* x, int64_t xi, int64_t xs, double* y,
                                  int64_t yi, int64_t ys, cudaStream_t st) {
    for (int j = 0; j < nv; j += kCsrMaxVec) {
        const double* xj = x + (int64_t)j * xs;
        double* yj = y + (int64_t)j * ys;
        const int w = nv - j < kCsrMaxVec ? nv - j : kCsrMaxVec;
        // one load per column for adjacent vectors whose group is aligned at every column
        const uintptr_t a = reinterpret_cast<uintptr_t>(xj);
        const int wide = xs != 1 ? 1 : (w == 4 && xi % 4 == 0 && a % 32 == 0) ? 4 : (w % 2 == 0 && xi % 2 == 0 && a % 16 == 0) ? 2 : 1;
        if (w == 4 && wide == 4)
            csr_pass<4, 4>(A, xj, xi, xs, yj, yi, ys, st);
        else if (w == 4 && wide == 2)
            csr_pass<4, 2>(A, xj, xi, xs, yj, yi, ys, st);
        else if (w == 4)
            csr_pass<4, 1>(A, xj, xi, xs, yj, yi, ys, st);
        else if (w == 3)
            csr_pass<3, 1>(A, xj, xi, xs, yj, yi, ys, st);
        else if (w == 2 && wide == 2)
            csr_pass<2, 2>(A, xj, xi, xs, yj, yi, ys, st);
        else if (w == 2)
            csr_pass<2, 1>(A, xj, xi, xs, yj, yi, ys, st);
        else
            csr_pass<1, 1>(A, xj, xi, xs, yj, yi, ys, st);
    }
    return cudaGetLastError();
}

cudaError_t launch_f64_to_f32(const double* a, float* b, int64_t n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_f64_to_f32<<<grid_for(n) > 4096 ? 4096 : grid_for(n), 256, 0, st>>>(a, b, n);
    return cudaGetLastError();
}

cudaError_t launch_f32_to_f64(const float* a, double* b, int64_t n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_f32_to_f64<<<grid_for(n) > 4096 ? 4096 : grid_for(n), 256, 0, st>>>(a, b, n);
    return cudaGetLastError();
}

}  // namespace sgdg

namespace sgdg {
cudaError_t launch_vlasov_points(const double* v, const double* F, const double* pt, int D, int64_t n, double* out,
                                 cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_vlasov_points<<<grid_for(n) > 4096 ? 4096 : grid_for(n), 256, 0, st>>>(v, F, pt, D, n, out);
    return cudaGetLastError();
}
}  // namespace sgdg

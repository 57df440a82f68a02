// csr_step.cu -- the plain form's stepping: FP64 CSR mat-vec (the closure body
// *(RHS, x) of src/pdes.jl:63) fused with the classical RK4 stage update, for
// one solve or for sets of solves that share the operator.
//
//  * k_csr_rk: rows binned by length (DevCSR.bin_*), a row of bin b summed by
//    2^b lanes with a few entries each (csr_lane_entries); every block of the
//    grid serves one bin.  NV solves go through a row together: a matrix entry
//    is loaded once and meets the set's interleaved values in one 16- or
//    32-byte load.  Bounds: large operators the FP64 pipe (2 operations per
//    clock and SM, the additions of the lane reduction and of the stage update
//    among them), small ones the latency of four dependent launches per step.
//    For the second the launches are programmatic dependents (pdl_wait): a
//    launch's blocks come up and fetch their row pointers, columns and values
//    while the launch before it still runs, and wait for it only before the
//    vectors.  200 steps of the 2D wave k=3 n=5 from host to host took 6.34 ms
//    with one solve at a time, the whole operator and plain launches, 1.94 ms
//    now; 60 steps of the 4D advection k=2 n=6 5.89 -> 1.42 ms; 3 steps of 48
//    3D waves k=3 n=7 11.8 -> 3.2 ms (0.94 ms per step, of which the FP64 pipe
//    needs 0.75).
//  * k_rk_segments, k_rk_long_rows: rows longer than A.split, one warp per
//    segment, then the segment partials of each row in order and the update.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "bounds.cuh"
#include "csr.cuh"
#include "engine.h"
#include "rk.cuh"

namespace sgdg {

struct CsrRK {  // stage update of the RK4 epilogue: k = A uin, then rk_stage
    double* acc;
    double* uout;
    double dt, hdt, dt6;
    int stage;
    int write_u;     // stage 4 also stores the new state to uout (the next step's input when it is not y)
    int* nonfinite;  // set to 1 when a stage result is not finite (may be null)
};

// Programmatic dependent launch: waits until the launches this one depends on
// have completed and their writes are visible, then lets the next launch come
// up.  Everything read before it (the operator) was written before those
// launches.  The vectors read after it are plain loads: another launch wrote
// them after this one's blocks came up, so they are not read-only for its
// lifetime.
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// 256-bit load (sm_100 and later); p 32-byte aligned
__device__ __forceinline__ void ld_v4(const double* p, double& a, double& b, double& c, double& d) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a), "=d"(b), "=d"(c), "=d"(d) : "l"(p) : "memory");
}

// the values of a set of NV interleaved vectors at one column
template <int NV>
__device__ __forceinline__ void set_gather(const double* x, int64_t col, double (&v)[NV]) {
    if constexpr (NV == 4) {
        ld_v4(x + col * 4, v[0], v[1], v[2], v[3]);
    } else if constexpr (NV == 2) {
        const double2 t = __ldca(reinterpret_cast<const double2*>(x + col * 2));
        v[0] = t.x;
        v[1] = t.y;
    } else {
        v[0] = __ldca(x + col);
    }
}

// entries a lane fetches ahead of the vectors (and before pdl_wait)
constexpr int kCsrAhead = 4;
struct CsrAhead {
    int c[kCsrAhead];  // column, -1 past the end
    double v[kCsrAhead];
};
template <int VS>
__device__ __forceinline__ void csr_fetch(const DevCSR& A, int64_t p, int64_t e, CsrAhead& t) {
#pragma unroll
    for (int u = 0; u < kCsrAhead; u++) {
        const int64_t q = p + u * VS;
        t.c[u] = -1;
        t.v[u] = 0.0;
        if (q < e) {
            t.c[u] = __ldg(A.col + q);
            t.v[u] = __ldg(A.val + q);
            if (!SGDG_IN(t.c[u], A.m)) t.c[u] = 0;  // debug build: counted, read column 0 instead
        }
    }
}

// s[j] = the row with entries [b, e) times vector j, summed over VS lanes: the
// entries b + lane, b + lane + VS, ... in order, the first of them in t already
// (b = e: zeros, but the lanes still take part); see csr_reduce for where the
// sums end up.  The order does not depend on NV, so a solve's result is the
// same alone and beside others.  The whole warp runs to its longest row, so
// that the additions past it are skipped by a branch: predicated off, they
// would still take their turn on the FP64 pipe.
template <int VS, int NV>
__device__ __forceinline__ void row_sum(const DevCSR& A, int64_t b, int64_t e, CsrAhead& t, const double* x, int lane,
                                        double (&s)[NV]) {
#pragma unroll
    for (int j = 0; j < NV; j++) s[j] = 0.0;
    const int most = __reduce_max_sync(0xffffffffu, (int)(e - b));
    int64_t p = b + lane;
    for (int done = 0; done < most; done += kCsrAhead * VS) {
        double xv[kCsrAhead][NV];
#pragma unroll
        for (int u = 0; u < kCsrAhead; u++)
            if (t.c[u] >= 0) set_gather<NV>(x, t.c[u], xv[u]);
        CsrAhead next;  // the entries after these, while the gathers are on their way
        p += kCsrAhead * VS;
        csr_fetch<VS>(A, p, e, next);
#pragma unroll
        for (int u = 0; u < kCsrAhead; u++) {
            if (done + u * VS >= most) break;
            if (t.c[u] >= 0) {
#pragma unroll
                for (int j = 0; j < NV; j++) s[j] = fma(t.v[u], xv[u][j], s[j]);
            }
        }
        t = next;
    }
    csr_reduce<VS, NV>(s, lane);
}

// RK4 stage update of one element: k its right-hand side, y its state, acc and
// uout at element `o` of the scratch vectors
__device__ __forceinline__ void csr_rk_update(const CsrRK& rk, double k, double* y, int64_t o) {
    double yy = *y, aa = rk.stage == 1 ? 0.0 : rk.acc[o], un;
    rk_stage(rk.stage, rk.dt, rk.hdt, rk.dt6, k, yy, aa, un);
    if (rk.stage == 4)
        *y = yy;
    else
        rk.acc[o] = aa;
    if (rk.stage != 4 || rk.write_u) rk.uout[o] = un;
    if (rk.nonfinite && (__double2hiint(un) & 0x7ff00000) == 0x7ff00000) *rk.nonfinite = 1;
}

// the rows of bin `bin`, 2^bin = VS lanes each; nv of the NV solves are stored,
// solve j's state at y + j A.m
template <int VS, int NV>
__device__ __forceinline__ void rk_bin(const DevCSR& A, int bin, int64_t rb, const double* x, double* y,
                                       const CsrRK& rk, int nv) {
    const int64_t t = (rb - A.bin_block[bin]) * blockDim.x + threadIdx.x;
    const int64_t idx = t / VS, first = A.bin_first[bin];
    const int lane = int(t % VS);
    int64_t row = idx < A.bin_first[bin + 1] - first ? (int64_t)__ldg(A.bin_rows + first + idx) : -1;
    if (row >= 0 && !SGDG_IN(row, A.m)) row = -1;
    int64_t b = 0, e = 0;
    if (row >= 0) {
        b = __ldg(A.rowptr + row);
        e = __ldg(A.rowptr + row + 1);
    }
    CsrAhead ahead;
    csr_fetch<VS>(A, b + lane, e, ahead);
    pdl_wait();
    double s[NV];
    row_sum<VS, NV>(A, b, e, ahead, x, lane, s);
    bool stores;
    const int owner = csr_owner<VS, NV>(lane, stores);
    if (row < 0 || !stores) return;
    if (owner >= 0) {
        if (owner < nv) csr_rk_update(rk, s[0], y + row + owner * A.m, row * NV + owner);
    } else {
#pragma unroll
        for (int j = 0; j < NV; j++)
            if (j < nv) csr_rk_update(rk, s[j], y + row + j * A.m, row * NV + j);
    }
}

// Sets of NV solves sharing A: set g's vectors (interleaved x, acc and uout,
// and the states one after another) start at g NV A.m.  Block b is (row block,
// set): the sets go in groups of `group`, and within a group the set index
// runs fastest, so the group's passes over a row block run side by side and
// read its matrix entries from L2 while the group's vectors stay there too (A
// is streamed once per group instead of once per set).
struct CsrSets {
    int64_t count;
    int group;
    int last;  // solves of the last set
};

template <int NV>
__global__ void __launch_bounds__(256, NV == 1 ? 6 : 4)
    k_csr_rk(DevCSR A, const double* x, double* y, CsrRK rk, CsrSets q) {
    int64_t rb = blockIdx.x, g = 0;
    if (q.count > 1) {
        const int64_t nrb = A.bin_block[kCsrBins], b = blockIdx.x, full = q.count / q.group, fb = full * nrb * q.group;
        if (b < fb) {
            const int64_t grp = b / (nrb * q.group), r = b - grp * nrb * q.group;
            rb = r / q.group;
            g = grp * q.group + r % q.group;
        } else {
            const int64_t tail = q.count - full * q.group, r = b - fb;
            rb = r / tail;
            g = full * q.group + r % tail;
        }
        const int64_t o = g * NV * A.m;
        x += o;
        y += o;
        rk.acc += o;
        rk.uout += o;
    }
    const int nv = g + 1 == q.count ? q.last : NV;
    int bin = 0;
    while (bin + 1 < kCsrBins && rb >= A.bin_block[bin + 1]) bin++;
    switch (bin) {
        case 0: rk_bin<1, NV>(A, 0, rb, x, y, rk, nv); break;
        case 1: rk_bin<2, NV>(A, 1, rb, x, y, rk, nv); break;
        case 2: rk_bin<4, NV>(A, 2, rb, x, y, rk, nv); break;
        case 3: rk_bin<8, NV>(A, 3, rb, x, y, rk, nv); break;
        case 4: rk_bin<16, NV>(A, 4, rb, x, y, rk, nv); break;
        default: rk_bin<32, NV>(A, 5, rb, x, y, rk, nv); break;
    }
}

// one warp per segment of a long row
__global__ void __launch_bounds__(256) k_rk_segments(DevCSR A, const double* x) {
    const int64_t seg = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    int64_t b = 0, e = 0;
    if (seg < A.nseg) {
        b = __ldg(A.seg_begin + seg);
        e = __ldg(A.seg_end + seg);
    }
    CsrAhead ahead;
    csr_fetch<32>(A, b + lane, e, ahead);
    pdl_wait();
    double s[1];
    row_sum<32, 1>(A, b, e, ahead, x, lane, s);
    if (seg < A.nseg && lane == 0) A.partial[seg] = s[0];
}

// one thread per long row: the row's segment partials in order, then the update
__global__ void k_rk_long_rows(DevCSR A, double* y, CsrRK rk) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    if (i >= A.nlong) return;
    double s = 0.0;
    for (int q = A.long_seg[i]; q < A.long_seg[i + 1]; q++) s += A.partial[q];
    const int64_t row = A.long_row[i];
    if (!SGDG_IN(row, A.m)) return;
    csr_rk_update(rk, s, y + row, row);
}

SGDG_BOUNDS_READER(step_bounds_violations)

// ------------------------------------------------------------ launchers ----
static int grid_for(int64_t threads) {
    int64_t b = (threads + 255) / 256;
    return (int)(b > (1LL << 30) ? (1LL << 30) : (b < 1 ? 1 : b));
}

// a launch that may come up while the one before it in the stream still runs
// (its kernel calls pdl_wait before it touches what that one writes)
template <class... P, class... Q>
static void launch_dependent(void (*kernel)(P...), int64_t blocks, cudaStream_t st, Q... args) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)blocks);
    c.blockDim = dim3(256);
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    (void)cudaLaunchKernelEx(&c, kernel, P(args)...);  // the caller reads the error with cudaGetLastError
}

cudaError_t launch_csr_rk4(const DevCSR& A, const double* uin, double* y, double* acc, double* uout, double dt,
                           int stage, int* nonfinite, cudaStream_t st) {
    const CsrRK rk{acc, uout, dt, 0.5 * dt, dt / 6.0, stage, 0, nonfinite};
    if (A.bin_block[kCsrBins] > 0)
        launch_dependent(k_csr_rk<1>, A.bin_block[kCsrBins], st, A, uin, y, rk, CsrSets{1, 1, 1});
    if (A.nlong > 0) {
        launch_dependent(k_rk_segments, grid_for(A.nseg * 32), st, A, uin);
        launch_dependent(k_rk_long_rows, grid_for(A.nlong), st, A, y, rk);
    }
    return cudaGetLastError();
}

// u[(g * len + i) * NV + j] = y[(g * NV + j) * len + i]: solve g NV + j of the
// states y, one after another, into interleaved sets (zeros past the last)
template <int NV>
__global__ void k_interleave(const double* __restrict__ y, double* __restrict__ u, int64_t len, int64_t nb) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, g = blockIdx.y;
    if (i >= len) return;
    double v[NV];
#pragma unroll
    for (int j = 0; j < NV; j++) v[j] = g * NV + j < nb ? y[(g * NV + j) * len + i] : 0.0;
#pragma unroll
    for (int j = 0; j < NV; j++) u[(g * len + i) * NV + j] = v[j];
}

// solves that go through a row together, given nb of them
int plain_set_size(const DevCSR& A, int64_t nb) { return A.nlong > 0 || nb < 2 ? 1 : nb == 2 ? 2 : kCsrMaxVec; }

// sets per group of the batched row kernel: 4 sets of 4 solves of the 3D k=3
// n=7 wave keep their vectors in L2 while they share A's rows
constexpr int kPlainSetGroup = 4;

template <int NV>
static void rk4_sets(const DevCSR& A, int64_t nb, double* y, double* acc, double* u0, double* u1, double dt, int stage,
                     int* nonfinite, cudaStream_t st) {
    const int64_t len = A.m, ng = (nb + NV - 1) / NV, nrb = A.bin_block[kCsrBins];
    const double* uin = stage % 2 ? u0 : u1;
    const int64_t most = std::max<int64_t>(1, ((int64_t(1) << 31) - 1) / std::max<int64_t>(nrb, 1));
    for (int64_t g = 0; g < ng && nrb > 0; g += most) {
        const int64_t n = std::min(most, ng - g), o = g * NV * len;
        const CsrRK rk{acc + o, (stage % 2 ? u1 : u0) + o, dt, 0.5 * dt, dt / 6.0, stage, 1, nonfinite};
        launch_dependent(k_csr_rk<NV>, nrb * n, st, A, uin + o, y + o, rk,
                         CsrSets{n, kPlainSetGroup, g + n == ng ? int(nb - (ng - 1) * NV) : NV});
    }
}

// nsteps RK4 steps of nb solves y' = A y that share A, their states one after
// another (solve s at y + s A.m).  A set of plain_set_size solves goes through
// a row together: the stage inputs and accumulators are interleaved, so a
// matrix entry is loaded once per set and meets a column's values in one
// load.  nv is plain_set_size or 1; acc, u0 and u1 hold whole sets of A.m
// numbers a solve, and with nv > 1 u0 holds the interleaved states on entry
// (launch_plain_interleave) and on return.
cudaError_t launch_plain_steps(const DevCSR& A, int nv, int64_t nb, double* y, double* acc, double* u0, double* u1,
                               double dt, int64_t nsteps, int* nonfinite, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    for (int64_t i = 0; i < nsteps && e == cudaSuccess; i++) {
        for (int stage = 1; stage <= 4 && e == cudaSuccess; stage++) {
            if (nv == 1) {
                for (int64_t s = 0; s < nb && e == cudaSuccess; s++) {
                    const int64_t o = s * A.m;
                    const double* in = stage == 1 ? y : stage == 3 ? u1 : u0;
                    e = launch_csr_rk4(A, in + o, y + o, acc + o, (stage == 2 ? u1 : u0) + o, dt, stage, nonfinite, st);
                }
                continue;
            }
            if (nv == 2)
                rk4_sets<2>(A, nb, y, acc, u0, u1, dt, stage, nonfinite, st);
            else
                rk4_sets<4>(A, nb, y, acc, u0, u1, dt, stage, nonfinite, st);
            e = cudaGetLastError();
        }
    }
    return e;
}

cudaError_t launch_plain_interleave(const DevCSR& A, int nv, int64_t nb, const double* y, double* u0,
                                    cudaStream_t st) {
    if (nv == 1 || A.m == 0) return cudaSuccess;
    const int64_t ng = (nb + nv - 1) / nv;
    for (int64_t g = 0; g < ng; g += 65535) {
        const int64_t n = std::min<int64_t>(65535, ng - g), o = g * nv * A.m;
        const dim3 grid((unsigned)((A.m + 255) / 256), (unsigned)n);
        if (nv == 2)
            k_interleave<2><<<grid, 256, 0, st>>>(y + o, u0 + o, A.m, nb - g * nv);
        else
            k_interleave<4><<<grid, 256, 0, st>>>(y + o, u0 + o, A.m, nb - g * nv);
    }
    return cudaGetLastError();
}

}  // namespace sgdg

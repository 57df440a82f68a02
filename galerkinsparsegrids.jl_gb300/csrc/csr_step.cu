// csr_step.cu -- the plain form's stepping: FP64 sparse mat-vec (the closure
// body *(RHS, x) of src/pdes.jl:63) fused with the classical RK4 stage update,
// for one solve or for sets of solves that share the operator, and the sweeps
// of the Vlasov right-hand side (src/pdes.jl:174-192).
//
//  * k_csr_rk: a row of bin b summed by 2^b lanes with a few entries each
//    (csr_lane_entries); every block of the grid serves one bin.  NV solves go
//    through a row together: a matrix entry is loaded once and meets the set's
//    interleaved values in one 16- or 32-byte load.  The stepping operators are
//    in slices (DevSliced: rows sorted by length, a warp's entries adjacent),
//    whole ones (DevCSR) in rows.
//  * k_rk_segments, k_rk_long_rows: rows longer than A.split, one warp per
//    segment, then the segment partials of each row in order and the update.
//  * k_derivatives, k_sweep, k_sweep_points, k_points: the P derivatives of a
//    phase-space vector; a transform along one dimension or a few for P
//    interleaved vectors or one; the products at the points, with the last
//    transform or alone.
//
// Bounds: large operators the FP64 pipe (2 operations per clock and SM, the
// additions of the lane reduction and of the stage update among them), small
// ones the latency of four dependent launches per step (Vlasov: up to 4 (4P + 2)).
// For the second the launches are programmatic dependents (pdl_wait): a
// launch's blocks come up and fetch their rows, columns and values while the
// launch before it still runs, and wait for it only before the vectors.
//
// Measured, from host to host: 200 steps of the 2D wave k=3 n=5 6.34 -> 1.84 ms
// against one solve at a time with the whole operator and plain launches; 60
// steps of the 4D advection k=2 n=6 5.89 -> 1.21 ms; 3 steps of 48 3D waves k=3
// n=7 11.8 -> 2.6 ms (0.87 ms per step, of which the FP64 pipe needs 0.74).
// In slices against rows: the single 3D wave 46.9 -> 38.1 us per step, 256 of
// them 4.80 -> 4.49 ms, the Vlasov step below 810 -> 634 us.  Vlasov 2x2v k=2
// n=8: 2595 -> 540 us per step against the assembled transforms, of which the
// FP64 pipe needs 240 and about 150 are the latency of 56 launches; n=5 296 ->
// 104 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

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
    int* nonfinite;  // one per solve: set to 1 when a stage result of its is not finite (not read with FLAGS = false)
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

// the values of NV adjacent vectors at one element
template <int NV>
__device__ __forceinline__ void set_gather(const double* x, double (&v)[NV]) {
    if constexpr (NV == 4) {
        ld_v4(x, v[0], v[1], v[2], v[3]);
    } else if constexpr (NV == 2) {
        const double2 t = __ldca(reinterpret_cast<const double2*>(x));
        v[0] = t.x;
        v[1] = t.y;
    } else {
        v[0] = __ldca(x);
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

// s[j] = the row with entries [b, e) times vector j (element i of the set at
// x + i stride), summed over VS lanes: the
// entries b + lane, b + lane + VS, ... in order, the first of them in t already
// (b = e: zeros, but the lanes still take part); see csr_reduce for where the
// sums end up.  The order does not depend on NV, so a solve's result is the
// same alone and beside others.  The whole warp runs to its longest row, so
// that the additions past it are skipped by a branch: predicated off, they
// would still take their turn on the FP64 pipe.
template <int VS, int NV>
__device__ __forceinline__ void row_sum(const DevCSR& A, int64_t b, int64_t e, CsrAhead& t, const double* x, int lane,
                                        int64_t stride, double (&s)[NV]) {
#pragma unroll
    for (int j = 0; j < NV; j++) s[j] = 0.0;
    const int most = __reduce_max_sync(0xffffffffu, (int)(e - b));
    int64_t p = b + lane;
    for (int done = 0; done < most; done += kCsrAhead * VS) {
        double xv[kCsrAhead][NV];
#pragma unroll
        for (int u = 0; u < kCsrAhead; u++)
            if (t.c[u] >= 0) set_gather<NV>(x + t.c[u] * stride, xv[u]);
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

__device__ __forceinline__ bool not_finite(double x) { return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000; }

// RK4 stage update of one element: k its right-hand side, yy its state and aa its
// accumulator (from y and acc[o]), which go back there and uout[o]; its solve's flag
// is rk.nonfinite[j]
template <bool FLAGS>
__device__ __forceinline__ void csr_rk_update(const CsrRK& rk, double k, double yy, double aa, double* y, int64_t o,
                                              int j) {
    double un;
    rk_stage(rk.stage, rk.dt, rk.hdt, rk.dt6, k, yy, aa, un);
    if (rk.stage == 4)
        *y = yy;
    else
        rk.acc[o] = aa;
    if (rk.stage != 4 || rk.write_u) rk.uout[o] = un;
    if (FLAGS && not_finite(un)) rk.nonfinite[j] = 1;
}

// Block rb's rows, 2^bin lanes each: out.one(row, j, sum) by the lane that
// holds vector j's sum, or out.all(row, sums) where one lane holds them all; what
// the lane needs for that besides is loaded before the sum (out.fetch), so that
// its latency passes under the gathers.
template <int VS, int NV, class Out>
__device__ __forceinline__ void bin_rows(const DevCSR& A, int bin, int64_t rb, const double* x, int64_t stride,
                                         const Out& out) {
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
    bool stores;
    const int owner = csr_owner<VS, NV>(lane, stores);
    typename Out::Fetched f;
    if (row >= 0 && stores) out.fetch(row, owner, f);
    double s[NV];
    row_sum<VS, NV>(A, b, e, ahead, x, lane, stride, s);
    if (row < 0 || !stores) return;
    if (owner >= 0)
        out.one(row, owner, s[0], f);
    else
        out.all(row, s, f);
}

// the same for slices
template <int VS, int NV, class Out>
__device__ __forceinline__ void bin_rows(const DevSliced& A, int64_t rb, const double* x, int64_t stride,
                                         const Out& out) {
    const int64_t slice = rb * kSliceWarps + (threadIdx.x >> 5);
    const int l32 = threadIdx.x & 31;
    int64_t row = __ldg(A.rows + slice * 32 + l32);
    const int64_t first = __ldg(A.base + slice);
    const int n = (int)(__ldg(A.base + slice + 1) - first);
    if (row >= 0 && !SGDG_IN(row, A.m)) row = -1;
    const int32_t* col = A.col + first * 32 + l32;
    const double* val = A.val + first * 32 + l32;
    auto fetch = [&](int u0, CsrAhead& t) {
#pragma unroll
        for (int u = 0; u < kCsrAhead; u++) {
            t.c[u] = -1;
            t.v[u] = 0.0;
            if (u0 + u < n) {  // the same for the whole warp
                t.c[u] = __ldg(col + (u0 + u) * 32);
                t.v[u] = __ldg(val + (u0 + u) * 32);
                if (t.c[u] >= 0 && !SGDG_IN(t.c[u], A.m)) t.c[u] = -1;
            }
        }
    };
    CsrAhead t;
    fetch(0, t);
    pdl_wait();
    const int lane = l32 % VS;
    bool stores;
    const int owner = csr_owner<VS, NV>(lane, stores);
    typename Out::Fetched f;
    if (row >= 0 && stores) out.fetch(row, owner, f);
    double s[NV];
#pragma unroll
    for (int j = 0; j < NV; j++) s[j] = 0.0;
    for (int u0 = 0; u0 < n; u0 += kCsrAhead) {
        double xv[kCsrAhead][NV];
#pragma unroll
        for (int u = 0; u < kCsrAhead; u++)
            if (t.c[u] >= 0) set_gather<NV>(x + t.c[u] * stride, xv[u]);
        CsrAhead next;
        fetch(u0 + kCsrAhead, next);
#pragma unroll
        for (int u = 0; u < kCsrAhead; u++) {
            if (u0 + u >= n) break;
            if (t.c[u] >= 0) {
#pragma unroll
                for (int j = 0; j < NV; j++) s[j] = fma(t.v[u], xv[u][j], s[j]);
            }
        }
        t = next;
    }
    csr_reduce<VS, NV>(s, lane);
    if constexpr (Out::kTogether && ((NV == 4 && VS >= 4) || (NV == 2 && VS >= 2))) {
        // the row's sums to its first lane (csr_owner's lanes)
        const double mine = s[0];
#pragma unroll
        for (int j = 0; j < NV; j++)
            s[j] = __shfl_sync(0xffffffffu, mine,
                               NV == 4 ? (j & 2 ? VS / 2 : 0) + (j & 1 ? VS / 4 : 0) : (j & 1 ? VS / 2 : 0), VS);
        if (row >= 0 && lane == 0) out.all(row, s, f);
        return;
    }
    if (row < 0 || !stores) return;
    if (owner >= 0)
        out.one(row, owner, s[0], f);
    else
        out.all(row, s, f);
}

template <int NV, class Out>
__device__ __forceinline__ void block_rows(const DevSliced& A, int64_t rb, const double* x, int64_t stride,
                                           const Out& out) {
    int bin = 0;
    while (bin + 1 < kCsrBins && rb >= A.bin_block[bin + 1]) bin++;
    switch (bin) {
        case 0: bin_rows<1, NV>(A, rb, x, stride, out); break;
        case 1: bin_rows<2, NV>(A, rb, x, stride, out); break;
        case 2: bin_rows<4, NV>(A, rb, x, stride, out); break;
        case 3: bin_rows<8, NV>(A, rb, x, stride, out); break;
        case 4: bin_rows<16, NV>(A, rb, x, stride, out); break;
        default: bin_rows<32, NV>(A, rb, x, stride, out); break;
    }
}

template <int NV, class Out>
__device__ __forceinline__ void block_rows(const DevCSR& A, int64_t rb, const double* x, int64_t stride, const Out& out) {
    int bin = 0;
    while (bin + 1 < kCsrBins && rb >= A.bin_block[bin + 1]) bin++;
    switch (bin) {
        case 0: bin_rows<1, NV>(A, 0, rb, x, stride, out); break;
        case 1: bin_rows<2, NV>(A, 1, rb, x, stride, out); break;
        case 2: bin_rows<4, NV>(A, 2, rb, x, stride, out); break;
        case 3: bin_rows<8, NV>(A, 3, rb, x, stride, out); break;
        case 4: bin_rows<16, NV>(A, 4, rb, x, stride, out); break;
        default: bin_rows<32, NV>(A, 5, rb, x, stride, out); break;
    }
}

// The stage update of nv of the NV solves of a set, solve j's state at y + j m.
// One solve, whose time is latency, fetches its state and accumulator before the
// sum (3D wave k=3 n=7 38.1 -> 35.8 us per step); sets, bound by the FP64 pipe,
// after it (256 of them 4.49 ms, 4.59 with the registers held across the sum).
// FLAGS: a result that is not finite raises its solve's flag.
template <int NV, bool FLAGS>
struct RkOut {
    static constexpr bool kTogether = false;
    struct Fetched {
        double y, acc;
    };
    const CsrRK& rk;
    double* y;
    int64_t m;
    int nv;
    int first;  // flag of solve 0
    __device__ __forceinline__ void load(int64_t row, int j, Fetched& f) const {
        f.y = y[row + j * m];
        f.acc = rk.stage != 1 ? rk.acc[row * NV + j] : 0.0;
    }
    __device__ __forceinline__ void fetch(int64_t row, int, Fetched& f) const {
        if constexpr (NV == 1) load(row, 0, f);
    }
    __device__ __forceinline__ void one(int64_t row, int j, double s, Fetched& f) const {
        if (j >= nv) return;
        if constexpr (NV > 1) load(row, j, f);
        csr_rk_update<FLAGS>(rk, s, f.y, f.acc, y + row + j * m, row * NV + j, NV == 1 ? 0 : first + j);
    }
    __device__ __forceinline__ void all(int64_t row, const double (&s)[NV], Fetched& f) const {
#pragma unroll
        for (int j = 0; j < NV; j++) one(row, j, s[j], f);
    }
};

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

// Only a pruned operator's steps are repeated where a value is not finite.
template <class Mat>
constexpr bool kFlags = std::is_same_v<Mat, DevSliced>;

template <int NV, class Mat>
__global__ void __launch_bounds__(256, NV == 1 ? 4 : 3)
    k_csr_rk(Mat A, const double* x, double* y, CsrRK rk, CsrSets q) {
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
    block_rows<NV>(A, rb, x, NV, RkOut<NV, kFlags<Mat>>{rk, y, A.m, g + 1 == q.count ? q.last : NV, (int)g * NV});
}

// One warp per segment of a long row, the sums in row_sum's order, in plain groups:
// segments are of one length but for the rows' last ones, and row_sum's predicated
// additions would take their turn on the FP64 pipe.  Groups of four, no look-ahead:
// 32 registers and 77 % of the warps active keep that pipe 86 % busy (DRAM 64 %).
// FEW: segments that are all resident at once are bound by their chain of loads
// (entries, gather, sum), so eight are on their way and the next eight fetched
// beside them.  us for 40 steps of the wave, row_sum, groups of four and FEW, with
// the segments: 2D k=3 n=9 12456, 13264, 11803 (54); 2D k=2 n=10 12768, 13898, 12060
// (4,560); 1D k=8 n=9 8053, 6954, 7548 (8,192); 2D k=4 n=9 5242, 4952, 5079 (32,736;
// 3 steps of 3).
constexpr int64_t kFewSegments = int64_t(kSMs) * 32;  // warps resident at FEW's 64 registers
template <bool FEW>
__global__ void __launch_bounds__(256) k_rk_segments(DevCSR A, const double* x) {
    constexpr int G = FEW ? 8 : 4;
    const int64_t seg = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    int64_t p = 0, e = 0;
    if (seg < A.nseg) {
        p = __ldg(A.seg_begin + seg) + lane;
        e = __ldg(A.seg_end + seg);
    }
    auto entry = [&](int64_t at, int& c, double& v) {
        c = __ldg(A.col + at);
        v = __ldg(A.val + at);
        if (!SGDG_IN(c, A.m)) c = 0;
    };
    int c[G];
    double v[G], s[1] = {0.0};
    auto group = [&](int (&gc)[G], double (&gv)[G]) {
#pragma unroll
        for (int u = 0; u < G; u++) entry(p + 32 * u, gc[u], gv[u]);
    };
    bool more = p + 32 * (G - 1) < e;
    if (more) group(c, v);
    pdl_wait();
    while (more) {
        double xv[G];
#pragma unroll
        for (int u = 0; u < G; u++) xv[u] = __ldca(x + c[u]);
        p += 32 * G;
        more = p + 32 * (G - 1) < e;
        int nc[G];
        double nv[G];
        if (FEW && more) group(nc, nv);
#pragma unroll
        for (int u = 0; u < G; u++) s[0] = fma(v[u], xv[u], s[0]);
        if (!more) break;
        if constexpr (FEW) {
#pragma unroll
            for (int u = 0; u < G; u++) {
                c[u] = nc[u];
                v[u] = nv[u];
            }
        } else {
            group(c, v);
        }
    }
    for (; p < e; p += 32) {
        int tc;
        double tv;
        entry(p, tc, tv);
        s[0] = fma(tv, __ldca(x + tc), s[0]);
    }
    csr_reduce<32, 1>(s, lane);
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
    csr_rk_update<false>(rk, s, y[row], rk.stage == 1 ? 0.0 : rk.acc[row], y + row, row, 0);
}

// NV adjacent vectors of an interleaved set (element i of vector j at
// y[i * stride + j]); for one vector a result that is not finite raises *nonfinite
// (the sweeps of several are followed by one that checks)
template <int NV>
struct SweepOut {
    static constexpr bool kTogether = false;
    struct Fetched {};
    double* y;
    int64_t stride;
    int* nonfinite;
    __device__ __forceinline__ void fetch(int64_t, int, Fetched&) const {}
    __device__ __forceinline__ void one(int64_t row, int j, double s, const Fetched&) const {
        y[row * stride + j] = s;
        if (NV == 1 && nonfinite && not_finite(s)) *nonfinite = 1;
    }
    __device__ __forceinline__ void all(int64_t row, const double (&s)[NV], const Fetched& f) const {
        double* p = y + row * stride;
        if constexpr (NV == 4)
            asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(s[0]), "d"(s[1]), "d"(s[2]), "d"(s[3])
                         : "memory");
        else if constexpr (NV == 2)
            *reinterpret_cast<double2*>(p) = make_double2(s[0], s[1]);
        else
            one(row, 0, s[0], f);
    }
};

// The point-basis combination of the Vlasov right-hand side (src/pdes.jl:
// 185-191) of the P = 2D transformed derivatives of a point q (x dimensions d <
// D, then p): -(sum_d v_d q_d) + sum_d F_d q_{D+d}, each sum left to right with
// separate roundings of products and sums.
template <int D>
__device__ __forceinline__ double point_product(const double* __restrict__ v, const double* __restrict__ F, int64_t n,
                                                int64_t i, const double (&q)[2 * D]) {
    double c1 = __dmul_rn(__ldg(v + i), q[0]), c2 = __dmul_rn(__ldg(F + i), q[D]);
#pragma unroll
    for (int d = 1; d < D; d++) {
        c1 = __dadd_rn(c1, __dmul_rn(__ldg(v + d * n + i), q[d]));
        c2 = __dadd_rn(c2, __dmul_rn(__ldg(F + d * n + i), q[D + d]));
    }
    return __dadd_rn(-c1, c2);
}

// The row block of one of a sweep's n blocks.  The slices ascend by row length;
// a grid of more blocks than are resident together takes the long rows first, so
// that short ones fill its end (8 steps of Vlasov 2x2v k=2 n=8 4885 -> 4511 us,
// k=3 n=6 4288 -> 4112); a smaller one starts them all at once and is faster in
// ascending order (k=2 n=7 2529 and 2343 us, n=6 1459 and 1279).
constexpr unsigned kSweepResident = kSMs * (768 / kSliceThreads);  // threads at 80 registers
__device__ __forceinline__ int sweep_block(int n) {
    return gridDim.x * gridDim.y > kSweepResident ? n - 1 - (int)blockIdx.x : (int)blockIdx.x;
}

// the products of a row's P = NV values
template <int NV>
struct PointsOut {
    static constexpr bool kTogether = true;
    const double *v, *F;
    double* out;
    int64_t n;
    struct Fetched {};
    __device__ __forceinline__ void fetch(int64_t, int, Fetched&) const {}
    __device__ __forceinline__ void one(int64_t, int, double, const Fetched&) const {}
    __device__ __forceinline__ void all(int64_t row, const double (&s)[NV], const Fetched&) const {
        out[row] = point_product<NV / 2>(v, F, n, row, s);
    }
};
template <int NV>
__global__ void __launch_bounds__(256, 3)
    k_sweep_points(DevSliced A, const double* x, const double* v, const double* F, double* out) {
    block_rows<NV>(A, sweep_block(gridDim.x), x, NV, PointsOut<NV>{v, F, out, A.m});
}

// One sweep y = T x of a transform along one dimension or a few, for sets of NV
// of `stride` interleaved vectors; blockIdx.y: the set.
template <int NV>
__global__ void __launch_bounds__(256, NV == 1 ? 4 : 3)
    k_sweep(DevSliced A, const double* x, double* y, int64_t stride, int* nonfinite) {
    const int64_t o = (int64_t)blockIdx.y * NV;
    block_rows<NV>(A, sweep_block(gridDim.x), x + o, stride, SweepOut<NV>{y + o, stride, nonfinite});
}

// One application y = A x with the pruned operator; an element of x that is not
// finite leaves `call` in *seen, for k_apply_whole
struct ApplyOut {
    static constexpr bool kTogether = false;
    const double* x;
    double* y;
    int* seen;
    int call;
    struct Fetched {
        double x;
    };
    __device__ __forceinline__ void fetch(int64_t row, int, Fetched& f) const { f.x = __ldca(x + row); }
    __device__ __forceinline__ void one(int64_t row, int, double s, const Fetched& f) const {
        y[row] = s;
        if (not_finite(f.x)) *seen = call;
    }
    __device__ __forceinline__ void all(int64_t row, const double (&s)[1], const Fetched& f) const { one(row, 0, s[0], f); }
};
__global__ void __launch_bounds__(256, 4) k_apply(DevSliced A, const double* x, double* y, int* seen, int call) {
    block_rows<1>(A, blockIdx.x, x, 1, ApplyOut{x, y, seen, call});
}

// y = A x with the whole operator, where this call's k_apply met an element of
// x that is not finite: the blocks share its row blocks, a warp takes a long row.
// left (null, or 0 before): the last block to leave clears *seen for the next
// replay of a captured call, which a memset before k_apply would do for 5 us more
// in each of them (12.3 us instead of 7.4, 3D k=3 n=7).
__global__ void __launch_bounds__(256)
    k_apply_whole(DevCSR A, const double* x, double* y, int* seen, int call, int* left) {
    pdl_wait();
    if (*reinterpret_cast<const volatile int*>(seen) != call) return;
    const SweepOut<1> out{y, 1, nullptr};
    for (int64_t rb = blockIdx.x; rb < A.bin_block[kCsrBins]; rb += gridDim.x) block_rows<1>(A, rb, x, 1, out);
    const int lane = threadIdx.x & 31;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < A.nlong;
         i += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int64_t row = A.long_row[i], b = A.rowptr[row], e = A.rowptr[row + 1];
        CsrAhead ahead;
        csr_fetch<32>(A, b + lane, e, ahead);
        double s[1];
        row_sum<32, 1>(A, b, e, ahead, x, lane, 1, s);
        if (lane == 0 && SGDG_IN(row, A.m)) y[row] = s[0];
    }
    if (!left) return;
    __syncthreads();  // every thread of the block has read *seen
    if (threadIdx.x == 0 && atomicAdd(left, 1) == (int)gridDim.x - 1) {
        *seen = 0;
        *left = 0;
    }
}

// The P derivatives of one vector, interleaved: y[i P + d] = (D_d x)_i; blockIdx.y: d.
struct DerivativeSet {
    DevSliced d[8];
};
__global__ void __launch_bounds__(256, 4)
    k_derivatives(const __grid_constant__ DerivativeSet S, const double* x, double* y, int64_t P) {
    const DevSliced& A = S.d[blockIdx.y];
    if ((int)blockIdx.x >= A.bin_block[kCsrBins]) {
        pdl_wait();
        return;
    }
    block_rows<1>(A, sweep_block(A.bin_block[kCsrBins]), x, 1, SweepOut<1>{y + blockIdx.y, P, nullptr});
}

// the same for P = 2D interleaved vectors pt[i 2D + d]
template <int D>
__global__ void k_points(const double* __restrict__ v, const double* __restrict__ F, const double* pt, int64_t n,
                         double* out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    if (i >= n) return;
    double q[2 * D];
#pragma unroll
    for (int d = 0; d < D; d++) {
        const double2 t = __ldca(reinterpret_cast<const double2*>(pt + i * 2 * D) + d);
        q[2 * d] = t.x;
        q[2 * d + 1] = t.y;
    }
    out[i] = point_product<D>(v, F, n, i, q);
}

__global__ void k_check_finite(const double* __restrict__ x, int64_t n, int* nonfinite) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        if (not_finite(x[i])) *nonfinite = 1;
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
static void launch_dependent(void (*kernel)(P...), dim3 grid, int threads, cudaStream_t st, Q... args) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = dim3((unsigned)threads);
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    (void)cudaLaunchKernelEx(&c, kernel, P(args)...);  // the caller reads the error with cudaGetLastError
}

template <class Mat>
constexpr int block_threads = std::is_same_v<Mat, DevSliced> ? kSliceThreads : 256;

template <class Mat>
static cudaError_t rk4_one(const Mat& A, const double* uin, double* y, const CsrRK& rk, cudaStream_t st) {
    if (kFlags<Mat> && !rk.nonfinite) return cudaErrorInvalidValue;
    if (A.bin_block[kCsrBins] > 0)
        launch_dependent(k_csr_rk<1, Mat>, A.bin_block[kCsrBins], block_threads<Mat>, st, A, uin, y, rk, CsrSets{1, 1, 1});
    if constexpr (std::is_same_v<Mat, DevCSR>)
        if (A.nlong > 0) {
            launch_dependent(A.nseg <= kFewSegments ? k_rk_segments<true> : k_rk_segments<false>, grid_for(A.nseg * 32), 256, st,
                             A, uin);
            launch_dependent(k_rk_long_rows, grid_for(A.nlong), 256, st, A, y, rk);
        }
    return cudaGetLastError();
}
cudaError_t launch_csr_rk4(const DevCSR& A, const double* uin, double* y, double* acc, double* uout, double dt,
                           int stage, int* nonfinite, cudaStream_t st) {
    return rk4_one(A, uin, y, CsrRK{acc, uout, dt, 0.5 * dt, dt / 6.0, stage, 0, nonfinite}, st);
}
cudaError_t launch_csr_rk4(const DevSliced& A, const double* uin, double* y, double* acc, double* uout, double dt,
                           int stage, int* nonfinite, cudaStream_t st) {
    return rk4_one(A, uin, y, CsrRK{acc, uout, dt, 0.5 * dt, dt / 6.0, stage, 0, nonfinite}, st);
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
int plain_set_size(const DevSliced&, int64_t nb) { return nb < 2 ? 1 : nb == 2 ? 2 : kCsrMaxVec; }
int plain_set_size(const DevCSR& A, int64_t nb) { return A.nlong > 0 || nb < 2 ? 1 : nb == 2 ? 2 : kCsrMaxVec; }

// sets per group of the batched row kernel: 4 sets of 4 solves of the 3D k=3
// n=7 wave keep their vectors in L2 while they share A's rows
constexpr int kPlainSetGroup = 4;

template <int NV, class Mat>
static void rk4_sets(const Mat& A, int64_t nb, double* y, double* acc, double* u0, double* u1, double dt, int stage,
                     int* nonfinite, cudaStream_t st) {
    const int64_t len = A.m, ng = (nb + NV - 1) / NV, nrb = A.bin_block[kCsrBins];
    const double* uin = stage % 2 ? u0 : u1;
    const int64_t most = std::max<int64_t>(1, ((int64_t(1) << 31) - 1) / std::max<int64_t>(nrb, 1));
    for (int64_t g = 0; g < ng && nrb > 0; g += most) {
        const int64_t n = std::min(most, ng - g), o = g * NV * len;
        const CsrRK rk{acc + o, (stage % 2 ? u1 : u0) + o, dt, 0.5 * dt, dt / 6.0, stage, 1,
                       nonfinite ? nonfinite + g * NV : nullptr};
        launch_dependent(k_csr_rk<NV, Mat>, (unsigned)(nrb * n), block_threads<Mat>, st, A, uin + o, y + o, rk,
                         CsrSets{n, kPlainSetGroup, g + n == ng ? int(nb - (ng - 1) * NV) : NV});
    }
}

// nsteps RK4 steps of nb solves y' = A y that share A, their states one after
// another (solve s at y + s A.m).  A set of plain_set_size solves goes through
// a row together: the stage inputs and accumulators are interleaved, so a
// matrix entry is loaded once per set and meets a column's values in one
// load.  nv is plain_set_size or 1; acc, u0 and u1 hold whole sets of A.m
// numbers a solve, nonfinite one flag a solve (null with a whole operator), and with
// nv > 1 u0 holds the interleaved states on entry (launch_plain_interleave) and on
// return.
template <class Mat>
static cudaError_t plain_steps(const Mat& A, int nv, int64_t nb, double* y, double* acc, double* u0, double* u1,
                               double dt, int64_t nsteps, int* nonfinite, cudaStream_t st) {
    cudaError_t e = kFlags<Mat> && !nonfinite ? cudaErrorInvalidValue : cudaSuccess;
    for (int64_t i = 0; i < nsteps && e == cudaSuccess; i++) {
        for (int stage = 1; stage <= 4 && e == cudaSuccess; stage++) {
            if (nv == 1) {
                for (int64_t s = 0; s < nb && e == cudaSuccess; s++) {
                    const int64_t o = s * A.m;
                    const double* in = stage == 1 ? y : stage == 3 ? u1 : u0;
                    e = launch_csr_rk4(A, in + o, y + o, acc + o, (stage == 2 ? u1 : u0) + o, dt, stage,
                                       nonfinite ? nonfinite + s : nullptr, st);
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

cudaError_t launch_plain_steps(const DevCSR& A, int nv, int64_t nb, double* y, double* acc, double* u0, double* u1,
                               double dt, int64_t nsteps, int* nonfinite, cudaStream_t st) {
    return plain_steps(A, nv, nb, y, acc, u0, u1, dt, nsteps, nonfinite, st);
}
cudaError_t launch_plain_steps(const DevSliced& A, int nv, int64_t nb, double* y, double* acc, double* u0, double* u1,
                               double dt, int64_t nsteps, int* nonfinite, cudaStream_t st) {
    return plain_steps(A, nv, nb, y, acc, u0, u1, dt, nsteps, nonfinite, st);
}

cudaError_t launch_plain_interleave(int64_t len, int nv, int64_t nb, const double* y, double* u0, cudaStream_t st) {
    if (nv == 1 || len == 0) return cudaSuccess;
    const int64_t ng = (nb + nv - 1) / nv;
    for (int64_t g = 0; g < ng; g += 65535) {
        const int64_t n = std::min<int64_t>(65535, ng - g), o = g * nv * len;
        const dim3 grid((unsigned)((len + 255) / 256), (unsigned)n);
        if (nv == 2)
            k_interleave<2><<<grid, 256, 0, st>>>(y + o, u0 + o, len, nb - g * nv);
        else
            k_interleave<4><<<grid, 256, 0, st>>>(y + o, u0 + o, len, nb - g * nv);
    }
    return cudaGetLastError();
}

// y = T x for P interleaved vectors (P = 1, or even; nonfinite for P = 1 only)
cudaError_t launch_sweep(const DevSliced& A, int P, const double* x, double* y, int* nonfinite, cudaStream_t st) {
    const unsigned nb = (unsigned)A.bin_block[kCsrBins];
    if (P > 1 && nonfinite) return cudaErrorInvalidValue;
    if (nb == 0) return cudaSuccess;
    if (P % 4 == 0)
        launch_dependent(k_sweep<4>, dim3(nb, P / 4), kSliceThreads, st, A, x, y, P, nonfinite);
    else if (P % 2 == 0)
        launch_dependent(k_sweep<2>, dim3(nb, P / 2), kSliceThreads, st, A, x, y, P, nonfinite);
    else
        launch_dependent(k_sweep<1>, dim3(nb, P), kSliceThreads, st, A, x, y, P, nonfinite);
    return cudaGetLastError();
}

// y = A x, P the pruned A; *seen is not `call` before, nor after where left is not null
cudaError_t launch_apply(const DevSliced& P, const DevCSR& A, const double* x, double* y, int* seen, int call, int* left,
                         cudaStream_t st) {
    if (P.bin_block[kCsrBins] == 0) return cudaSuccess;
    launch_dependent(k_apply, (unsigned)P.bin_block[kCsrBins], kSliceThreads, st, P, x, y, seen, call);
    launch_dependent(k_apply_whole, (unsigned)kSMs, 256, st, A, x, y, seen, call, left);
    return cudaGetLastError();
}

// y[i P + d] = (D_d x)_i for the P <= 8 operators D
cudaError_t launch_derivatives(const DevSliced* const* D, int P, const double* x, double* y, cudaStream_t st) {
    DerivativeSet S;
    int nb = 0;
    for (int d = 0; d < P; d++) {
        S.d[d] = *D[d];
        nb = std::max(nb, D[d]->bin_block[kCsrBins]);
    }
    for (int d = P; d < 8; d++) S.d[d] = *D[0];
    if (nb > 0) launch_dependent(k_derivatives, dim3((unsigned)nb, P), kSliceThreads, st, S, x, y, (int64_t)P);
    return cudaGetLastError();
}

// out = the products of the points of y = T x, x 2D interleaved vectors (D <= 2)
cudaError_t launch_sweep_points(const DevSliced& A, int D, const double* x, const double* v, const double* F, double* out,
                                cudaStream_t st) {
    const unsigned nb = (unsigned)A.bin_block[kCsrBins];
    if (nb > 0) launch_dependent(D == 1 ? k_sweep_points<2> : k_sweep_points<4>, nb, kSliceThreads, st, A, x, v, F, out);
    return cudaGetLastError();
}

// the products of 2D interleaved vectors (D = 3, 4)
cudaError_t launch_points(const double* v, const double* F, const double* pt, int D, int64_t n, double* out,
                          cudaStream_t st) {
    auto kernel = D == 3 ? k_points<3> : k_points<4>;
    if (n > 0) launch_dependent(kernel, (unsigned)grid_for(n), 256, st, v, F, pt, n, out);
    return cudaGetLastError();
}

cudaError_t launch_check_finite(const double* x, int64_t n, int* nonfinite, cudaStream_t st) {
    if (n > 0) k_check_finite<<<std::min(grid_for(n), 1024), 256, 0, st>>>(x, n, nonfinite);
    return cudaGetLastError();
}

}  // namespace sgdg

// capi.cu -- the C ABI of libsgdg (include/sgdg.h).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <set>
#include <string>
#include <vector>

#include "../../include/sgdg.h"
#include "device_util.h"
#include "engine.h"
#include "api_util.h"
#include "device_csr.h"
#include "mf_engine.h"
#include "sgdg_core.h"

namespace sgdg {

cudaError_t launch_csr_spmv(const DevCSR& A, const double* x, double* y, cudaStream_t st);
cudaError_t mf_bounds_violations(unsigned int* out, bool reset);
cudaError_t csr_bounds_violations(unsigned int* out, bool reset);
cudaError_t step_bounds_violations(unsigned int* out, bool reset);
cudaError_t asm_bounds_violations(unsigned int* out, bool reset);
cudaError_t launch_csr_rk4(const DevCSR& A, const double* uin, double* y, double* acc, double* uout, double dt,
                           int stage, int* nonfinite, cudaStream_t st);
cudaError_t launch_csr_rk4(const DevSliced& A, const double* uin, double* y, double* acc, double* uout, double dt,
                           int stage, int* nonfinite, cudaStream_t st);
int plain_set_size(const DevCSR& A, int64_t nb);
int plain_set_size(const DevSliced& A, int64_t nb);
cudaError_t launch_plain_steps(const DevCSR& A, int nv, int64_t nb, double* y, double* acc, double* u0, double* u1,
                               double dt, int64_t nsteps, int* nonfinite, cudaStream_t st);
cudaError_t launch_plain_steps(const DevSliced& A, int nv, int64_t nb, double* y, double* acc, double* u0, double* u1,
                               double dt, int64_t nsteps, int* nonfinite, cudaStream_t st);
cudaError_t launch_plain_interleave(int64_t len, int nv, int64_t nb, const double* y, double* u0, cudaStream_t st);
cudaError_t launch_csr_spmv_multi(const DevCSR& A, int nv, const double* x, int64_t xi, int64_t xs, double* y,
                                  int64_t yi, int64_t ys, cudaStream_t st);
cudaError_t launch_vlasov_points(const double* v, const double* F, const double* pt, int D, int64_t n, double* out,
                                 cudaStream_t st);
cudaError_t launch_sweep(const DevSliced& A, int P, const double* x, double* y, int* nonfinite, cudaStream_t st);
cudaError_t launch_apply(const DevSliced& P, const DevCSR& A, const double* x, double* y, int* seen, int call, int* left,
                         cudaStream_t st);
cudaError_t launch_derivatives(const DevSliced* const* D, int P, const double* x, double* y, cudaStream_t st);
cudaError_t launch_points(const double* v, const double* F, const double* pt, int D, int64_t n, double* out,
                          cudaStream_t st);
cudaError_t launch_sweep_points(const DevSliced& A, int D, const double* x, const double* v, const double* F, double* out,
                                cudaStream_t st);
cudaError_t launch_check_finite(const double* x, int64_t n, int* nonfinite, cudaStream_t st);
cudaError_t launch_wait_selftest(const int* ctr, int need, int* err, cudaStream_t st);
cudaError_t launch_convert_selftest(const double* x, int64_t n, unsigned long long* bad, cudaStream_t st);

static thread_local std::string g_err;
void set_error(const std::string& msg) { g_err = msg; }

// ------------------------------------------------------- plain form ----
}  // namespace sgdg

using namespace sgdg;

// ------------------------------------------------------------ handles ----
struct sgdg_op : LiveHandle, Spare {
    SparseIndex ix;
    std::shared_ptr<const DLF1D> dlf;
    int basis = SGDG_BASIS_HIER;  // SGDG_BASIS_POS: the 1D position-basis operators
    std::vector<std::unique_ptr<CSR>> dd;  // D_d, built on demand
    std::unique_ptr<CSR> lap, wave;
    std::map<int, std::unique_ptr<DeviceCSR>> dev;  // plain-form device copies by `which`
    std::map<int, std::unique_ptr<DeviceSliced>> step_dev;  // without the rounding of zeros (stepping)
    std::unique_ptr<DeviceAdvection> adv;
    std::map<int, int> refused;  // `which`: the budget (g_budget_set) that had no room for its pruned form
    static constexpr int kAdvection = INT32_MIN;  // adv, beside the selectors
    std::map<int, std::unique_ptr<MFEngine>> mf_apply;
    cudaStream_t stream = nullptr;

    const CSR& get(int which) {
        const int D = ix.D;
        if (basis == SGDG_BASIS_POS) {
            if (which != 1 && which != SGDG_OP_LAPLACIAN && which != SGDG_OP_WAVE_RHS)
                throw Error(SGDG_EINVAL, "operator selector must be 1, 0 (laplacian) or -1 (wave RHS)");
            if (!lap) {
                dd[0].reset(new CSR());
                lap.reset(new CSR());
                pos_operators(ix.k, ix.n, dd[0].get(), lap.get());
            }
            if (which == 1) return *dd[0];
            if (which == SGDG_OP_LAPLACIAN) return *lap;
            if (!wave) wave.reset(new CSR(wave_rhs(*lap)));
            return *wave;
        }
        if (which >= 1 && which <= D) {
            if (!dd[which - 1]) dd[which - 1].reset(new CSR(assemble_dd(ix, *dlf, which - 1)));
            return *dd[which - 1];
        }
        if (which == SGDG_OP_LAPLACIAN || which == SGDG_OP_WAVE_RHS) {
            if (!lap) {
                std::vector<const CSR*> v;
                for (int d = 1; d <= D; d++) v.push_back(&get(d));
                lap.reset(new CSR(spgemm_sum(v)));
            }
            if (which == SGDG_OP_LAPLACIAN) return *lap;
            if (!wave) wave.reset(new CSR(wave_rhs(*lap)));
            return *wave;
        }
        throw Error(SGDG_EINVAL, "operator selector must be 1..D, 0 (laplacian) or -1 (wave RHS)");
    }
    const DevCSR& device(int which) {
        auto it = dev.find(which);
        if (it == dev.end())
            it = dev.emplace(which, basis == SGDG_BASIS_POS ? to_device(get(which), stream)
                                                            : gpu_operator(ix, *dlf, which, stream))
                     .first;
        return it->second->d;
    }
    // The operator the plain evolvers step with: without the entries that hold
    // only the rounding of a zero (line_tables), which are most of the stored
    // ones (3D k=3 n=7: 191 entries per row of the Laplacian, 41 of them
    // nonzero).  They do carry NaN and infinities from one row to another, so
    // a run that meets one is repeated with the whole operator (plain_run).
    // The whole operators' own rounding grows with k and eightfold per level in a
    // Laplacian (relative L2 of what the two give for sums of Fourier modes: 3D
    // k=3 n=7 1e-10, 2D k=4 n=7 3e-10, n=9 6e-9; after 200 steps of the wave 2D
    // k=4 n=7 4e-11, n=9 7e-10; after 200 of the advection at most 5e-13).  Nearly
    // all of that is the whole operator's (200 steps of the wave 2D k=4 n=9 against
    // 64 bits: whole 7.1e-10, pruned 3.4e-13), but it is what the reference gives:
    // second derivatives and applications are pruned where the results stay within
    // 1e-10 or so of it, and finer grids keep the whole operator and its time.
    static constexpr int kPruneWave = 11, kPruneApply = 10;  // k + n at most
    bool prunes(bool second, int most) const {
        return basis == SGDG_BASIS_HIER && ix.k <= kPruneMaxK && (!second || ix.k + ix.n <= most);
    }
    // Without room for it, now or earlier under the same budget: null, and the
    // caller goes on with the whole operator.  The caller holds a Use.
    const DevSliced* stepping(int which) {
        auto it = step_dev.find(which);
        if (it == step_dev.end()) {
            std::unique_ptr<DeviceSliced> S;
            if (!build_pruned(which, [&] { S = gpu_step_operator(ix, *dlf, which, stream); })) return nullptr;
            it = step_dev.emplace(which, std::move(S)).first;
        }
        return &it->second->d;
    }
    // sum_d s[d] D_d, as stepping()
    const DevSliced* advection(const double* s) {
        if (!adv && !build_pruned(kAdvection, [&] { adv = gpu_advection(ix, *dlf, stream); })) return nullptr;
        CK(adv->scale(ix.D, s, stream));
        return &adv->A.d;
    }
    template <class Build>
    bool build_pruned(int which, Build&& build) {
        const auto f = refused.find(which);
        if (f != refused.end() && f->second == g_budget_set.load()) return false;
        try {
            build();
            return true;
        } catch (const Error& e) {
            if (e.code != SGDG_ENOMEM_BUDGET) throw;
            refused[which] = g_budget_set.load();
            return false;
        }
    }
    // what is there beside the whole operators, but for captured calls'
    bool drop_spare() override {
        bool any = adv != nullptr;
        if (adv) refused[kAdvection] = g_budget_set.load();
        adv.reset();
        for (auto it = step_dev.begin(); it != step_dev.end();) {
            if (!dev.count(it->first) || in_graphs.count(it->first)) {
                ++it;
                continue;
            }
            refused[it->first] = g_budget_set.load();
            it = step_dev.erase(it);
            any = true;
        }
        return any;
    }
    // Applications of an operator of kApplyPruned entries or more go through the
    // pruned one (us per application, whole and pruned: Laplacian 2D k=3 n=7, 1.3
    // M entries, 8.3 and 8.9; 4D k=2 n=6, 1.6 M, 10.3 and 8.9; 3D k=3 n=6, 2.2 M,
    // 11.5 and 9.1; 3D k=3 n=7, 8.8 M, 28.3 and 9.0; below 9 the time is the
    // caller's, two launches for one; building both takes the first application
    // 14.7 ms instead of 10.0 for the last of them, 5.7 instead of 3.4 for the 4D
    // one), and where an element of x is not finite through the whole one after it
    // (k_apply_whole).  Each call leaves its number in a word of its own among
    // kApplyCalls: calls on other streams may still be in flight.  A captured call,
    // whose number is the same in every replay, has two words for good (the second
    // for k_apply_whole to clear the first) and keeps the pruned operator there; with
    // a budget set, without the operator, or after kApplyCalls of them, it is
    // captured with the whole one.
    static constexpr int64_t kApplyPruned = 3 << 19;
    static constexpr int kApplyCalls = 1024;
    DevBuf apply_seen;  // the calls' words, then the pairs of captured calls
    int apply_call = 0, apply_captured = 0;
    std::set<int> in_graphs;  // `which` of pruned operators that captured calls use
    cudaError_t apply(int which, const double* x, double* y, cudaStream_t st) {
        const DevCSR& A = whole(which);
        if (!prunes(true, kPruneApply) || A.nnz < kApplyPruned) return launch_csr_spmv(A, x, y, st);
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        const cudaError_t e = st ? cudaStreamIsCapturing(st, &cap) : cudaSuccess;  // (the legacy stream never is)
        if (e != cudaSuccess) return e;
        Use use(*this);
        if (cap != cudaStreamCaptureStatusNone) {
            if (g_budget.load() > 0 || !apply_seen.p || !step_dev.count(which) || apply_captured == kApplyCalls)
                return launch_csr_spmv(A, x, y, st);
            in_graphs.insert(which);
            int* seen = apply_seen.as<int>() + kApplyCalls + 2 * apply_captured++;
            return launch_apply(step_dev.at(which)->d, A, x, y, seen, 1, seen + 1, st);
        }
        const DevSliced* P = stepping(which);
        if (P && !apply_seen.p && !build_pruned(which, [&] {
                DevBuf seen(3 * sizeof(int) * kApplyCalls);
                CK(cudaMemsetAsync(seen.p, 0, seen.bytes, stream));
                CK(cudaStreamSynchronize(stream));
                apply_seen = std::move(seen);
            }))
            P = nullptr;
        if (!P) return launch_csr_spmv(A, x, y, st);
        apply_call = apply_call == INT32_MAX ? 1 : apply_call + 1;
        return launch_apply(*P, A, x, y, apply_seen.as<int>() + apply_call % kApplyCalls, apply_call, nullptr, st);
    }
    // the whole operator, the pruned one making room for it where there is none
    const DevCSR& whole(int which) {
        const auto it = dev.find(which);
        if (it != dev.end()) return it->second->d;
        Use use(*this);
        try {
            return device(which);
        } catch (const Error& e) {
            if (e.code != SGDG_ENOMEM_BUDGET) throw;
            if (step_dev.erase(which) + drop_spare() == 0) throw;  // (no call of it was captured without the whole one)
        }
        return device(which);
    }
    ~sgdg_op() {
        retire();
        dev.clear();
        step_dev.clear();
        adv.reset();
        mf_apply.clear();
        if (stream) cudaStreamDestroy(stream);
    }
};

// ----------------------------------------------------------- Vlasov ----
// Operators of vlasov_evolve (src/pdes.jl:131-227) for D space dimensions:
// phase space of P = 2D dimensions (x_1..x_D, p_1..p_D), grad_matrix(P), the
// four nodal transforms and the velocity points v_d = n2p m2n (2 p_d - 1).
// The device operators are assembled on the GPU when the handle first goes
// there; the host copies of the transforms are built only when asked for
// (export), and the velocity points with the device transforms when a GPU
// is present, else with the host ones.
//
// The right-hand side is stepped as sweeps: a D-dimensional transform is the
// product of its 1D map along each dimension in turn, exactly, because the 1D
// maps are triangular in the level (no intermediate leaves the sparse grid).
// 2x2v k=2 n=8 multiplies 15 + 18 + 8 + 20 entries per coefficient that way
// where the assembled transforms hold 147 + 120 + 12 + 244, and the derivatives
// go without the rounding of zeros (22 entries instead of 50).  The assembled
// operators (whole_rhs) are built and used when a run meets a value that is not
// finite, which they spread over more rows, or where the sweeps have no room;
// once they are there, the sweeps give way to an allocation that needs theirs.
struct sgdg_vlasov : LiveHandle, Spare {
    int D = 0, P = 0, k = 0, n = 0;
    SparseIndex ix;
    std::shared_ptr<const DLF1D> dlf;
    mutable std::unique_ptr<CSR> T[4];    // m2n, n2p, p2n, n2m on the host, built on request
    mutable std::vector<double> v_point;  // D x N, built on request
    mutable bool have_vpoint = false;
    // sweep[w]: transform w in turn along the dimensions, one or a few at a time; deriv[d]: D_d
    std::vector<std::unique_ptr<DeviceSliced>> sweep[4];
    std::unique_ptr<DeviceSliced> deriv[8];
    // the assembled operators, built on request
    std::vector<std::unique_ptr<DeviceCSR>> dDs;
    std::unique_ptr<DeviceCSR> dT[4];
    DevBuf vpt, F, t, s, c, z;  // t, s: P vectors each, interleaved (t[i * P + d])
    DevBuf p;                   // P vectors for the assembled operators
    DevBuf flag;                // a result was not finite
    cudaStream_t stream = nullptr;
    int refused = -1;           // the budget (g_budget_set) that had no room for the sweeps
    ~sgdg_vlasov() {
        retire();
        if (stream) cudaStreamDestroy(stream);
    }
    const CSR& host_transform(int w) const {
        if (!T[w]) T[w].reset(new CSR(transform_dd(ix, transform_1d(k, n, w))));
        return *T[w];
    }
    // modal coefficients of 2 p_d - 1: 1/sqrt(3) on mode 2 along dimension D + d
    // of the first block (the tensor product with 1), src/pdes.jl:166-172
    std::vector<double> v_modal(int d) const {
        std::vector<double> vm(ix.N, 0.0);
        vm[(size_t)std::pow((double)k, (double)(D + d))] = 1.0 / std::sqrt(3.0);
        return vm;
    }
    void vpoint_host() const {  // n2p m2n on the host
        const int64_t N = ix.N;
        v_point.assign((size_t)D * N, 0.0);
        std::vector<double> tmp(N), pt(N);
        auto spmv = [&](const CSR& A, const std::vector<double>& x, std::vector<double>& y) {
            for (int64_t i = 0; i < A.m; i++) {
                double acc = 0.0;
                for (int64_t q = A.rowptr[i]; q < A.rowptr[i + 1]; q++) acc += A.val[q] * x[A.col[q]];
                y[i] = acc;
            }
        };
        for (int d = 0; d < D; d++) {
            spmv(host_transform(0), v_modal(d), tmp);
            spmv(host_transform(1), tmp, pt);
            std::copy(pt.begin(), pt.end(), v_point.begin() + (size_t)d * N);
        }
        have_vpoint = true;
    }
    void to_gpu() {  // the caller holds a Use
        if (flag.p) return;
        require_gpu();
        if (!stream) CK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
        const bool sweeps = have_sweeps();
        if (!sweeps) build_whole();
        const size_t b = sizeof(double) * (size_t)ix.N;
        if (!have_vpoint) {  // n2p m2n with the device transforms
            DevBuf x(b), y(b);
            v_point.assign((size_t)D * ix.N, 0.0);
            for (int d = 0; d < D; d++) {
                const std::vector<double> vm = v_modal(d);
                CK(cudaMemcpyAsync(x.p, vm.data(), b, cudaMemcpyHostToDevice, stream));
                double *from = x.as<double>(), *to = y.as<double>();
                for (int w : {0, 1}) {
                    if (sweeps) {
                        CK(transform(w, sweep[w].size(), 1, from, to));
                    } else {
                        CK(launch_csr_spmv(dT[w]->d, from, to, stream));
                        std::swap(from, to);
                    }
                }
                CK(cudaMemcpyAsync(v_point.data() + (size_t)d * ix.N, from, b, cudaMemcpyDeviceToHost, stream));
                CK(cudaStreamSynchronize(stream));
            }
            have_vpoint = true;
        }
        vpt = upload(v_point, stream);
        F.alloc(b * D);
        t.alloc(b * P);
        s.alloc(b * P);
        c.alloc(b);
        z.alloc(b);
        CK(cudaStreamSynchronize(stream));
        flag.alloc(sizeof(int));
    }
    // Dimensions a sweep of transform w takes at once.  More at once multiply
    // more entries (the product of the dimensions' rows instead of their sum) in
    // fewer launches of about 2.5 us each.  points -> nodal has at most 3 entries
    // per row and dimension: four at once are 12 entries instead of 7.7 (2x2v k=2
    // n=8).  modal -> nodal and nodal -> points take pairs up to 128 K values (us per step,
    // one by one and in pairs: 2x2v k=2 n=5 173 and 125, n=6 219 and 214; k=3 n=5,
    // 179 K values, 347 and 369), nodal -> modal, whose coarsest rows span a line
    // or for a pair a plane, up to 16 K coefficients in planes of 1 K (2x2v k=2 n=5
    // 184 and 173; n=6, 24 K, 220 and 226); in two dimensions, where a pair's
    // rows reach the whole grid, all three up to such a plane (1x1v k=2 n=6 82 and
    // 64, k=3 n=5 86 and 70; k=2 n=8, a plane of 5 K, 100 and 139).
    int at_once(int w) const {
        if (w == TRANSFORM_POINTS_TO_NODAL) return 4;
        if (w == TRANSFORM_NODAL_TO_MODAL)
            return ix.N <= 16 << 10 && make_index(2, k, n, ix.scheme).N <= 1 << 10 ? 2 : 1;
        return ix.N * P <= (P == 2 ? 4 << 10 : 128 << 10) ? 2 : 1;
    }
    void build_sweeps() {
        if (!sweep[3].empty()) return;
        std::vector<std::unique_ptr<DeviceSliced>> s[4];
        for (int d = 0; d < P; d++) deriv[d] = gpu_step_operator(ix, *dlf, d + 1, stream);
        for (int w = 0; w < 4; w++) {
            const CSR T1 = transform_1d(k, n, w);
            const LineTables T = line_tables(T1, k, n + 1);
            const int step = at_once(w);
            for (int d = 0; d < P; d += step)
                s[w].push_back(step == 1 ? gpu_line_operator(ix, T, d, stream)
                                         : gpu_partial_transform(ix, T1, ((1u << std::min(step, P - d)) - 1) << d, stream));
        }
        for (int w = 0; w < 4; w++) sweep[w] = std::move(s[w]);
    }
    void drop_sweeps() {
        for (auto& d : deriv) d.reset();
        for (auto& s : sweep) s.clear();
    }
    // builds the sweeps where there is room for them; false: the assembled
    // operators are to be used
    bool have_sweeps() {
        if (!sweep[3].empty()) return true;
        if (refused == g_budget_set.load()) return false;
        try {
            build_sweeps();
            return true;
        } catch (const Error& e) {
            if (e.code != SGDG_ENOMEM_BUDGET) throw;
        }
        drop_sweeps();
        refused = g_budget_set.load();
        return false;
    }
    bool drop_spare() override {
        if (!p.p || sweep[3].empty()) return false;
        drop_sweeps();
        refused = g_budget_set.load();
        return true;
    }
    // the first `count` sweeps of transform w of nv interleaved vectors, from x;
    // the result is in x, y is scratch (the two pointers change places)
    cudaError_t transform(int w, size_t count, int nv, double*& x, double*& y) {
        cudaError_t e = cudaSuccess;
        for (size_t i = 0; i < count && e == cudaSuccess; i++, std::swap(x, y))
            e = launch_sweep(sweep[w][i]->d, nv, x, y, nullptr, stream);
        return e;
    }
    // all sweeps of n2m but the last, of p2n (-sum_d v_d .* n2p m2n Dx_d u + sum_d
    // F_d .* n2p m2n Dp_d u): the P derivatives, interleaved, each transform's
    // sweeps on all P of them at a time, the point products (with the last sweep
    // for P <= 4) and the sweeps back.  last_sweep takes `result`.
    cudaError_t sweep_rhs(const double* u, double** result) {
        double *tt = t.as<double>(), *ss = s.as<double>(), *cc = c.as<double>(), *zz = z.as<double>();
        const double *v = vpt.as<double>(), *f = F.as<double>();
        const DevSliced* D_[8];
        for (int d = 0; d < P; d++) D_[d] = &deriv[d]->d;
        const size_t np = sweep[1].size();
        cudaError_t e = launch_derivatives(D_, P, u, tt, stream);
        if (e == cudaSuccess) e = transform(0, sweep[0].size(), P, tt, ss);
        if (e == cudaSuccess) e = transform(1, P <= 4 ? np - 1 : np, P, tt, ss);
        if (e == cudaSuccess)
            e = P <= 4 ? launch_sweep_points(sweep[1][np - 1]->d, D, tt, v, f, cc, stream)
                       : launch_points(v, f, tt, D, ix.N, cc, stream);
        if (e == cudaSuccess) e = transform(2, sweep[2].size(), 1, cc, zz);
        if (e == cudaSuccess) e = transform(3, sweep[3].size() - 1, 1, cc, zz);
        *result = cc;
        return e;
    }
    const DevSliced& last_sweep() const { return sweep[3].back()->d; }
    // the assembled operators and their scratch; the sweeps make room for them where there is none
    void build_whole() {
        if (p.p) return;
        auto build = [&] {
            // the phase-space derivatives keep 8 entries per lane, like the transforms they feed
            // (at 32 the plain step took 2.67 ms against 2.60)
            for (int d = (int)dDs.size(); d < P; d++)
                dDs.push_back(gpu_operator(ix, *dlf, d + 1, stream, kCsrLaneEntriesMulti));
            for (int w = 0; w < 4; w++)
                if (!dT[w]) dT[w] = gpu_transform(ix, transform_1d(k, n, w), stream);
            p.alloc(sizeof(double) * (size_t)ix.N * P);
            CK(cudaStreamSynchronize(stream));
        };
        try {
            build();
        } catch (const Error& e) {
            if (e.code != SGDG_ENOMEM_BUDGET || sweep[3].empty()) throw;
            drop_sweeps();
            refused = g_budget_set.load();
            build();
        }
    }
    // z = p2n (-sum_d v_d .* n2p m2n Dx_d u + sum_d F_d .* n2p m2n Dp_d u):
    // the P derivatives, interleaved (the P values of one coefficient share a
    // sector), then each transform on all P of them in one pass over its
    // matrix, the point products, and p2n
    cudaError_t whole_rhs(const double* u) {
        const int64_t N = ix.N;
        double *tt = t.as<double>(), *ss = s.as<double>(), *pp = p.as<double>();
        cudaError_t e = cudaSuccess;
        for (int d = 0; d < P && e == cudaSuccess; d++)
            e = launch_csr_spmv_multi(dDs[d]->d, 1, u, 1, 0, tt + d, P, 0, stream);
        if (e == cudaSuccess) e = launch_csr_spmv_multi(dT[0]->d, P, tt, P, 1, ss, P, 1, stream);
        if (e == cudaSuccess) e = launch_csr_spmv_multi(dT[1]->d, P, ss, P, 1, pp, P, 1, stream);
        if (e == cudaSuccess) e = launch_vlasov_points(vpt.as<double>(), F.as<double>(), pp, D, N, c.as<double>(), stream);
        if (e == cudaSuccess) e = launch_csr_spmv(dT[2]->d, c.as<double>(), z.as<double>(), stream);
        return e;
    }
};

// RK4 steps of the plain form: launched as they are, or `per` steps captured as a
// graph and replayed where the run is long enough to pay for the capture (launches
// are programmatic dependents either way).  A graph costs a call about 110 us for
// 32 launches and saves 0.5 to 1 us per step (us per step, launched and replayed:
// 2D wave k=3 n=5 9.26 and 8.76, 4D advection k=2 n=6 20.1 and 19.1, 3D wave k=3
// n=7 36.4 and 35.8; Vlasov 2x2v k=2 n=8, whose step alone is captured, 676 and
// 634 with 72 launches, 0.2 ms).
constexpr int64_t kGraphSteps = 256;       // of 4 launches
constexpr int64_t kGraphStepsVlasov = 16;  // of 20 to 100
class StepGraph {
   public:
    StepGraph(int64_t per, bool use) : per_(per), use_(use) {}
    StepGraph(const StepGraph&) = delete;
    StepGraph& operator=(const StepGraph&) = delete;
    ~StepGraph() {
        if (exec_) cudaGraphExecDestroy(exec_);
    }
    // launches nsteps steps on st (never the legacy stream), steps(n) launching n of them
    template <class Steps>
    void run(int64_t nsteps, cudaStream_t st, Steps&& steps) {
        if (use_ && nsteps >= per_ && !exec_) capture(st, steps);
        for (; exec_ && nsteps >= per_; nsteps -= per_) CK(cudaGraphLaunch(exec_, st));
        CK(steps(nsteps));
    }

   private:
    template <class Steps>
    void capture(cudaStream_t st, Steps&& steps) {
        cudaGraph_t g = nullptr;
        CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        const cudaError_t e = steps(per_);
        const cudaError_t e2 = cudaStreamEndCapture(st, &g);
        if (e != cudaSuccess || e2 != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            throw Error(SGDG_ECUDA, std::string("capture: ") + cudaGetErrorString(e != cudaSuccess ? e : e2));
        }
        const cudaError_t e3 = cudaGraphInstantiate(&exec_, g, 0);
        cudaGraphDestroy(g);
        if (e3 != cudaSuccess) {
            exec_ = nullptr;
            throw Error(SGDG_ECUDA, std::string("instantiate: ") + cudaGetErrorString(e3));
        }
    }
    const int64_t per_;
    const bool use_;
    cudaGraphExec_t exec_ = nullptr;
};

struct sgdg_batch : LiveHandle {
    MFEngine eng;  // its destructor frees device memory only, never touches a stream
    cudaStream_t own = nullptr;
    ~sgdg_batch() {
        if (own) cudaStreamDestroy(own);
    }
};

static void copy_str(const std::string& s, char* buf, size_t len) {
    if (!buf || len == 0) return;
    size_t n = std::min(len - 1, s.size());
    std::memcpy(buf, s.data(), n);
    buf[n] = 0;
}

static cudaStream_t op_stream(sgdg_op* op) {
    require_gpu();
    if (!op->stream) CK(cudaStreamCreateWithFlags(&op->stream, cudaStreamNonBlocking));
    return op->stream;
}

// Point weights of the matrix-free Vlasov right-hand side: term d < Dx is
// -v_d .* (x-derivative), term Dx + d is F_d .* (p-derivative); each weight as
// an FP32 (hi, lo) pair (a rounded weight would perturb the operator
// systematically).  Layout: hi of all 2 Dx terms, then lo.
static std::vector<float> vlasov_weights(const SparseIndex& ix, int Dx, const double* F) {
    const int64_t N = ix.N;
    const int P = 2 * Dx;
    const std::vector<double> v = vlasov_velocity_points(ix, Dx);
    std::vector<float> w((size_t)2 * P * N);
    for (int t = 0; t < P; t++)
        for (int64_t e = 0; e < N; e++) {
            const double x = t < Dx ? -v[(size_t)t * N + e] : F[(size_t)(t - Dx) * N + e];
            const float hi = (float)x;
            w[(size_t)t * N + e] = hi;
            w[((size_t)P + t) * N + e] = (float)(x - (double)hi);
        }
    return w;
}

// nodal transforms: the D-dimensional restricted Kronecker product of a 1D map
static CSR build_transform(int D, int k, int n, int scheme, int which) {
    if (which < 0 || which > 3) throw Error(SGDG_EINVAL, "transform must be 0..3 (m2n, n2p, p2n, n2m)");
    return transform_dd(make_index(D, k, n, scheme), transform_1d(k, n, which));
}

static void export_csr(const CSR& A, int64_t* rowptr, int32_t* col, double* val) {
    std::memcpy(rowptr, A.rowptr.data(), sizeof(int64_t) * A.rowptr.size());
    if (A.nnz()) {
        std::memcpy(col, A.col.data(), sizeof(int32_t) * A.col.size());
        std::memcpy(val, A.val.data(), sizeof(double) * A.val.size());
    }
}

extern "C" {

// ---------------------------------------------------- nodal transforms ----

int sgdg_version(char* buf, size_t len) {
    copy_str("sgdg 0.1 (sm_103a)", buf, len);
    return SGDG_OK;
}

int sgdg_last_error(char* buf, size_t len) {
    copy_str(g_err, buf, len);
    return SGDG_OK;
}

int sgdg_get_size(int D, int k, int n, int scheme, int64_t* N) {
    API_BEGIN
    NEED(N);
    *N = make_index(D, k, n, scheme).N;
    API_END
}

int sgdg_index_map(int D, int k, int n, int scheme, int32_t* level, int32_t* cell, int32_t* mode) {
    API_BEGIN
    NEED(level);
    NEED(cell);
    NEED(mode);
    SparseIndex ix = make_index(D, k, n, scheme);
    int64_t j = 0;
    for (int b = 0; b < ix.nlev; b++) {
        const int* L = &ix.levels[(size_t)b * D];
        for (int64_t cl = 0; cl < ix.lev_cells[b]; cl++)
            for (int64_t ml = 0; ml < ix.kD; ml++) {
                int64_t c = cl, m = ml;
                for (int q = 0; q < D; q++) {
                    level[j * D + q] = L[q];
                    int64_t nc = ncells(L[q]);
                    cell[j * D + q] = int32_t(c % nc) + 1;
                    c /= nc;
                    mode[j * D + q] = int32_t(m % k) + 1;
                    m /= k;
                }
                j++;
            }
    }
    API_END
}

int sgdg_dg_coeffs(int k, double* out) {
    API_BEGIN
    NEED(out);
    const Basis1D& B = basis(k);
    std::memcpy(out, B.dg.data(), sizeof(double) * B.dg.size());
    API_END
}

static CSR dlf_csr(int k, int n) {
    auto op = dlf1d(k, n);
    CSR A;
    A.m = A.n = int64_t(k) << n;
    A.rowptr.assign(A.m + 1, 0);
    for (int rb = 0; rb < op->nblocks; rb++)
        for (int i = 0; i < k; i++) {
            int64_t row = (int64_t)rb * k + i;
            for (int p = op->rowptr[rb]; p < op->rowptr[rb + 1]; p++)
                for (int j = 0; j < k; j++) {
                    A.col.push_back(op->colblk[p] * k + j);
                    A.val.push_back(op->val[(size_t)p * k * k + i * k + j]);
                }
            A.rowptr[row + 1] = (int64_t)A.col.size();
        }
    return A;
}

int sgdg_dlf_1d_nnz(int k, int n, int64_t* nnz) {
    API_BEGIN
    NEED(nnz);
    basis(k);
    auto op = dlf1d(k, n);
    *nnz = (int64_t)op->colblk.size() * k * k;
    API_END
}

int sgdg_dlf_1d_export(int k, int n, int64_t* rowptr, int32_t* col, double* val) {
    API_BEGIN
    NEED(rowptr);
    NEED(col);
    NEED(val);
    CSR A = dlf_csr(k, n);
    std::memcpy(rowptr, A.rowptr.data(), sizeof(int64_t) * A.rowptr.size());
    std::memcpy(col, A.col.data(), sizeof(int32_t) * A.col.size());
    std::memcpy(val, A.val.data(), sizeof(double) * A.val.size());
    API_END
}

int sgdg_op_create(int D, int k, int n, int scheme, sgdg_op** out) {
    API_BEGIN
    NEED(out);
    *out = nullptr;
    if (n < 2) throw Error(SGDG_EINVAL, "n must be >= 2");
    auto op = std::make_unique<sgdg_op>();
    op->ix = make_index(D, k, n, scheme);
    op->dlf = dlf1d(k, n);
    op->dd.resize(D);
    *out = op.release();
    API_END
}

int sgdg_op_create_1d(int k, int n, int basis, sgdg_op** out) {
    API_BEGIN
    NEED(out);
    *out = nullptr;
    if (basis != SGDG_BASIS_HIER && basis != SGDG_BASIS_POS)
        throw Error(SGDG_EINVAL, "basis must be SGDG_BASIS_HIER (0) or SGDG_BASIS_POS (1)");
    if (n < 2) throw Error(SGDG_EINVAL, "n must be >= 2");
    auto op = std::make_unique<sgdg_op>();
    op->ix = make_index(1, k, n, SGDG_SCHEME_SPARSE);
    op->dlf = dlf1d(k, n);
    op->dd.resize(1);
    op->basis = basis;
    *out = op.release();
    API_END
}

int sgdg_op_destroy(sgdg_op* op) {
    API_BEGIN
    delete op;
    API_END
}

int sgdg_op_size(const sgdg_op* op, int64_t* N) {
    API_BEGIN
    NEED(op);
    NEED(N);
    *N = op->ix.N;
    API_END
}

int sgdg_op_nnz(sgdg_op* op, int which, int64_t* nnz) {
    API_BEGIN
    NEED(op);
    NEED(nnz);
    *nnz = op->get(which).nnz();
    API_END
}

int sgdg_op_device_nnz(sgdg_op* op, int which, int64_t* nnz) {
    API_BEGIN
    NEED(op);
    NEED(nnz);
    op_stream(op);
    *nnz = op->whole(which).nnz;
    API_END
}

int sgdg_op_export_device_csr(sgdg_op* op, int which, int64_t* rowptr, int32_t* col, double* val) {
    API_BEGIN
    NEED(op);
    NEED(rowptr);
    NEED(col);
    NEED(val);
    cudaStream_t st = op_stream(op);
    op->whole(which);
    const CSR A = download_csr(*op->dev.at(which), st);
    std::memcpy(rowptr, A.rowptr.data(), sizeof(int64_t) * A.rowptr.size());
    std::memcpy(col, A.col.data(), sizeof(int32_t) * A.col.size());
    std::memcpy(val, A.val.data(), sizeof(double) * A.val.size());
    API_END
}

int sgdg_op_export_csr(sgdg_op* op, int which, int64_t* rowptr, int32_t* col, double* val) {
    API_BEGIN
    NEED(op);
    NEED(rowptr);
    NEED(col);
    NEED(val);
    const CSR& A = op->get(which);
    std::memcpy(rowptr, A.rowptr.data(), sizeof(int64_t) * A.rowptr.size());
    std::memcpy(col, A.col.data(), sizeof(int32_t) * A.col.size());
    std::memcpy(val, A.val.data(), sizeof(double) * A.val.size());
    API_END
}

static void apply_device_impl(sgdg_op* op, int which, int method, const double* x, double* y, cudaStream_t st) {
    if (method == SGDG_METHOD_PLAIN) {
        CK(op->apply(which, x, y, st));
        return;
    }
    if (method != SGDG_METHOD_MATFREE) throw Error(SGDG_EINVAL, "method must be PLAIN (0) or MATFREE (1)");
    if (op->basis != SGDG_BASIS_HIER) throw Error(SGDG_EUNSUPPORTED, "the matrix-free form is hierarchical only");
    if (!(which == SGDG_OP_LAPLACIAN || (which >= 1 && which <= op->ix.D)))
        throw Error(SGDG_EUNSUPPORTED, "matrix-free apply supports which = 1..D or 0 (laplacian)");
    auto it = op->mf_apply.find(which);
    if (it == op->mf_apply.end()) {
        auto eng = std::make_unique<MFEngine>(st);
        SolveSpec sp{};
        sp.kind = which == SGDG_OP_LAPLACIAN ? MF_KIND_WAVE : MF_KIND_ADVECT;
        sp.D = op->ix.D;
        sp.k = op->ix.k;
        sp.n = op->ix.n;
        sp.scheme = op->ix.scheme;
        sp.dt = 0.0;
        sp.apply = true;
        sp.apply_dim = which >= 1 ? which - 1 : -1;
        eng->add(sp, nullptr);
        it = op->mf_apply.emplace(which, std::move(eng)).first;
    }
    it->second->set_stream(st);
    it->second->apply(x, y);
}

int sgdg_apply(sgdg_op* op, int which, int method, const double* x, double* y) {
    API_BEGIN
    NEED(op);
    NEED(x);
    NEED(y);
    cudaStream_t st = op_stream(op);
    const int64_t len = which == SGDG_OP_WAVE_RHS ? 2 * op->ix.N : op->ix.N;
    DevBuf dx(sizeof(double) * len), dy(sizeof(double) * len);
    CK(cudaMemcpyAsync(dx.p, x, sizeof(double) * len, cudaMemcpyHostToDevice, st));
    apply_device_impl(op, which, method, dx.as<double>(), dy.as<double>(), st);
    CK(cudaMemcpyAsync(y, dy.p, sizeof(double) * len, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    dx.recycle();
    dy.recycle();
    API_END
}

int sgdg_apply_device(sgdg_op* op, int which, int method, const double* x_dev, double* y_dev, void* stream) {
    API_BEGIN
    NEED(op);
    NEED(x_dev);
    NEED(y_dev);
    require_gpu();
    apply_device_impl(op, which, method, x_dev, y_dev, (cudaStream_t)stream);
    API_END
}

static std::vector<int64_t> out_steps(int64_t nsteps, int nout) {
    std::vector<int64_t> s(nout);
    for (int i = 0; i < nout; i++) s[i] = (int64_t)((__int128)nsteps * i / (nout - 1));
    return s;
}

}  // extern "C"

// One evolution y' = A y from host to host; returns whether a stage result
// was not finite.
template <class Mat>
static bool plain_run(const Mat& A, const double* y0, int64_t len, double t0, double t1, int64_t nsteps, int nout,
                      double* times, double* states, cudaStream_t st) {
    const size_t b = sizeof(double) * (size_t)len;
    constexpr bool pruned = std::is_same_v<Mat, DevSliced>;  // to be repeated where a result is not finite
    DevBuf work(4 * b + (pruned ? sizeof(int) : 0));
    double* y = work.as<double>();
    double *acc = y + len, *u0 = y + 2 * len, *u1 = y + 3 * len;
    int* flag = pruned ? reinterpret_cast<int*>(y + 4 * len) : nullptr;
    if (flag) CK(cudaMemsetAsync(flag, 0, sizeof(int), st));
    CK(cudaMemcpyAsync(y, y0, b, cudaMemcpyHostToDevice, st));
    const double dt = (t1 - t0) / double(nsteps);
    const auto steps = out_steps(nsteps, nout);
    StepGraph graph(8, nsteps >= kGraphSteps);
    int64_t done = 0;
    int bad = 0;
    for (int i = 0; i < nout; i++) {
        graph.run(steps[i] - done, st, [&](int64_t n) { return launch_plain_steps(A, 1, 1, y, acc, u0, u1, dt, n, flag, st); });
        done = steps[i];
        CK(cudaMemcpyAsync(states + (size_t)i * len, y, b, cudaMemcpyDeviceToHost, st));
        if (times) times[i] = t0 + (t1 - t0) * double(steps[i]) / double(nsteps);
    }
    if (flag) CK(cudaMemcpyAsync(&bad, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    work.recycle();
    return bad != 0;
}

// The wave (a = null) or advection with velocity a, stepped with the pruned
// operator; with the whole one if a stage was not finite, or where there is no
// room for the pruned one and the vectors.
static void plain_evolve(sgdg_op* op, const double* a, const double* y0, int64_t len, double t0, double t1,
                         int64_t nsteps, int nout, double* times, double* states) {
    cudaStream_t st = op_stream(op);
    Spare::Use use(*op);
    std::vector<double> s;  // -sum_d a_d D_d
    for (int d = 0; a && d < op->ix.D; d++) s.push_back(-a[d]);
    const DevSliced* P = nullptr;
    if (op->prunes(a == nullptr, op->kPruneWave)) P = a ? op->advection(s.data()) : op->stepping(SGDG_OP_WAVE_RHS);
    try {
        if (P && !plain_run(*P, y0, len, t0, t1, nsteps, nout, times, states, st)) return;
    } catch (const Error& e) {
        if (e.code != SGDG_ENOMEM_BUDGET) throw;
    }
    auto run = [&] {
        if (a) {
            op->adv.reset();
            // assembled on the GPU (the same entries as add_scaled)
            const auto A = gpu_scaled_sum(op->ix, *op->dlf, s.data(), st);
            plain_run(A->d, y0, len, t0, t1, nsteps, nout, times, states, st);
        } else {
            plain_run(op->whole(SGDG_OP_WAVE_RHS), y0, len, t0, t1, nsteps, nout, times, states, st);
        }
    };
    try {
        run();
        return;
    } catch (const Error& e) {
        if (e.code != SGDG_ENOMEM_BUDGET || !op->drop_spare()) throw;
    }
    run();
}

// The scratch of nsteps RK4 steps of nb solves sharing A.
struct PlainScratch {
    DevBuf acc, u0, u1, flag;
    int nv;
    template <class Mat>
    PlainScratch(const Mat& A, int64_t nb, int nv_) : nv(nv_) {
        const size_t b = sizeof(double) * (size_t)((nb + nv - 1) / nv * nv * A.m);
        if (std::is_same_v<Mat, DevSliced>) flag.alloc(sizeof(int) * (size_t)nb);
        acc.alloc(b);
        u0.alloc(b);
        u1.alloc(b);
    }
    void recycle() {  // after run
        for (DevBuf* b : {&acc, &u0, &u1, &flag}) b->recycle();
    }
    // waits for the steps; with the pruned operator, which solves had a stage result
    // that was not finite (one int each)
    template <class Mat>
    std::vector<int> run(const Mat& A, int64_t nb, double* y, double dt, int64_t nsteps, cudaStream_t st) {
        std::vector<int> bad(flag.p ? (size_t)nb : 0);
        StepGraph graph(8, nsteps >= kGraphSteps);
        if (flag.p) CK(cudaMemsetAsync(flag.p, 0, sizeof(int) * bad.size(), st));
        CK(launch_plain_interleave(A.m, nv, nb, y, u0.as<double>(), st));
        graph.run(nsteps, st, [&](int64_t n) {
            return launch_plain_steps(A, nv, nb, y, acc.as<double>(), u0.as<double>(), u1.as<double>(), dt, n,
                                      flag.as<int>(), st);
        });
        if (flag.p) CK(cudaMemcpyAsync(bad.data(), flag.p, sizeof(int) * bad.size(), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        return bad;
    }
};

// Steps solves with the whole operator, in its own scratch.
static void plain_whole_steps(sgdg_op* op, int which, int64_t nsolves, double* y, double dt, int64_t nsteps,
                              cudaStream_t st) {
    const DevCSR& W = op->whole(which);
    std::unique_ptr<PlainScratch> work;
    for (int nv = plain_set_size(W, nsolves); !work;) {
        try {
            work.reset(new PlainScratch(W, nsolves, nv));
        } catch (const Error& e) {
            if (e.code != SGDG_ENOMEM_BUDGET || (nv == 1 && !op->drop_spare())) throw;
            nv = 1;
        }
    }
    work->run(W, nsolves, y, dt, nsteps, st);
    work->recycle();
}

// nsteps plain FP64 RK4 steps of nsolves solves y' = A y sharing operator
// `which`, states device-resident one after another.  The pruned operator
// needs the states of the call's start beside the scratch vectors, to repeat
// the steps of a solve with the whole one if a stage of its was not finite (the
// others' results stand: a solve's do not depend on its neighbours); without room
// for them, or for sets padded to whole ones, the whole operator steps the solves
// one by one from the start.
static void plain_batch_steps(sgdg_op* op, int which, int64_t nsolves, double* y, double dt, int64_t nsteps,
                              cudaStream_t st) {
    struct Own {  // work is captured and overlapped on a stream of its own where the caller gives none
        cudaStream_t s = nullptr;
        ~Own() {
            if (s) cudaStreamDestroy(s);
        }
    } own;
    cudaStream_t cs = st;
    if (cs == nullptr) {
        CK(cudaStreamCreateWithFlags(&own.s, cudaStreamNonBlocking));
        cs = own.s;
        CK(cudaStreamSynchronize(nullptr));
    }
    Spare::Use use(*op);
    const DevSliced* A = op->prunes(which < 1, op->kPruneWave) ? op->stepping(which) : nullptr;
    std::unique_ptr<PlainScratch> work;
    DevBuf keep;
    if (A) try {
            work.reset(new PlainScratch(*A, nsolves, plain_set_size(*A, nsolves)));
            keep.alloc(sizeof(double) * (size_t)(nsolves * A->m));
        } catch (const Error& e) {
            if (e.code != SGDG_ENOMEM_BUDGET) throw;
            work.reset();
        }
    if (!keep.p) return plain_whole_steps(op, which, nsolves, y, dt, nsteps, cs);
    CK(cudaMemcpyAsync(keep.p, y, keep.bytes, cudaMemcpyDeviceToDevice, cs));
    const std::vector<int> bad = work->run(*A, nsolves, y, dt, nsteps, cs);
    work->recycle();
    if (std::find(bad.begin(), bad.end(), 1) == bad.end()) return keep.recycle();
    const int64_t len = A->m;
    auto restore = [&](int64_t first, int64_t n) {
        CK(cudaMemcpyAsync(y + first * len, keep.as<double>() + first * len, sizeof(double) * (size_t)(n * len),
                           cudaMemcpyDeviceToDevice, cs));
    };
    bool fits = true;
    try {
        for (int64_t i = 0, n; i < nsolves; i += n) {
            for (n = 1; i + n < nsolves && bad[i + n] == bad[i];) n++;
            if (!bad[i]) continue;
            restore(i, n);
            plain_whole_steps(op, which, n, y + i * len, dt, nsteps, cs);
        }
    } catch (const Error& e) {
        if (e.code != SGDG_ENOMEM_BUDGET) throw;
        fits = false;  // beside the states of the call's start
    }
    if (!fits) restore(0, nsolves);
    CK(cudaStreamSynchronize(cs));
    keep.recycle();
    if (!fits) plain_whole_steps(op, which, nsolves, y, dt, nsteps, cs);
}

extern "C" {

static void mf_evolve(sgdg_op* op, int kind, const double* a, const double* y0, int64_t len, double t0, double t1,
                      int64_t nsteps, int nout, double* times, double* states) {
    if (op->basis != SGDG_BASIS_HIER) throw Error(SGDG_EUNSUPPORTED, "the matrix-free form is hierarchical only");
    cudaStream_t st = op_stream(op);
    MFEngine eng(st);
    SolveSpec sp{};
    sp.kind = kind;
    sp.D = op->ix.D;
    sp.k = op->ix.k;
    sp.n = op->ix.n;
    sp.scheme = op->ix.scheme;
    for (int d = 0; d < sp.D; d++) sp.a[d] = a ? a[d] : 0.0;
    sp.dt = (t1 - t0) / double(nsteps);
    sp.apply_dim = -1;
    int id = eng.add(sp, y0);
    auto steps = out_steps(nsteps, nout);
    int64_t done = 0;
    for (int i = 0; i < nout; i++) {
        eng.step(steps[i] - done);
        done = steps[i];
        eng.get_state(id, states + (size_t)i * len);
        if (times) times[i] = t0 + (t1 - t0) * double(steps[i]) / double(nsteps);
    }
    eng.recycle();
}

static void check_evolve_args(int64_t nsteps, int nout, double t0, double t1) {
    if (nsteps < 1) throw Error(SGDG_EINVAL, "nsteps must be >= 1");
    if (nout < 2) throw Error(SGDG_EINVAL, "nout must be >= 2");
    if (!(std::isfinite(t0) && std::isfinite(t1)) || t1 == t0) throw Error(SGDG_EINVAL, "need finite t0 != t1");
}

int sgdg_op_plain_steps_device(sgdg_op* op, int which, int64_t nsolves, double* y_dev, double dt, int64_t nsteps,
                               void* stream) {
    API_BEGIN
    NEED(op);
    NEED(y_dev);
    if (nsolves < 1) throw Error(SGDG_EINVAL, "nsolves must be >= 1");
    if (nsteps < 0) throw Error(SGDG_EINVAL, "nsteps must be >= 0");
    if (!std::isfinite(dt)) throw Error(SGDG_EINVAL, "dt must be finite");
    require_gpu();
    if (nsteps > 0) plain_batch_steps(op, which, nsolves, y_dev, dt, nsteps, (cudaStream_t)stream);
    API_END
}

int sgdg_debug_bounds(int* checked, int64_t* violations, int reset) {
    API_BEGIN
    NEED(checked);
    NEED(violations);
    *violations = 0;
#ifdef SGDG_DEBUG
    *checked = 1;
#else
    *checked = 0;
    return SGDG_OK;  // nothing is checked (or counted) in this build
#endif
    require_gpu();
    unsigned int v = 0;
    for (auto f : {mf_bounds_violations, csr_bounds_violations, step_bounds_violations, asm_bounds_violations}) {
        CK(f(&v, reset != 0));
        *violations += v;
    }
    API_END
}

int sgdg_wave_evolve(sgdg_op* op, const double* f0, const double* v0, double t0, double t1, int64_t nsteps, int nout,
                     int method, double* times, double* states) {
    API_BEGIN
    NEED(op);
    NEED(f0);
    NEED(v0);
    NEED(states);
    check_evolve_args(nsteps, nout, t0, t1);
    const int64_t N = op->ix.N;
    std::vector<double> y0(2 * N);
    std::memcpy(y0.data(), f0, sizeof(double) * N);
    std::memcpy(y0.data() + N, v0, sizeof(double) * N);
    if (method == SGDG_METHOD_PLAIN)
        plain_evolve(op, nullptr, y0.data(), 2 * N, t0, t1, nsteps, nout, times, states);
    else if (method == SGDG_METHOD_MATFREE)
        mf_evolve(op, MF_KIND_WAVE, nullptr, y0.data(), 2 * N, t0, t1, nsteps, nout, times, states);
    else
        throw Error(SGDG_EINVAL, "method must be PLAIN (0) or MATFREE (1)");
    API_END
}

int sgdg_advect_evolve(sgdg_op* op, const double* a, const double* f0, double t0, double t1, int64_t nsteps, int nout,
                       int method, double* times, double* states) {
    API_BEGIN
    NEED(op);
    NEED(a);
    NEED(f0);
    NEED(states);
    check_evolve_args(nsteps, nout, t0, t1);
    if (op->basis != SGDG_BASIS_HIER) throw Error(SGDG_EUNSUPPORTED, "advection is hierarchical only");
    const int64_t N = op->ix.N;
    if (method == SGDG_METHOD_PLAIN) {
        plain_evolve(op, a, f0, N, t0, t1, nsteps, nout, times, states);
    } else if (method == SGDG_METHOD_MATFREE) {
        mf_evolve(op, MF_KIND_ADVECT, a, f0, N, t0, t1, nsteps, nout, times, states);
    } else {
        throw Error(SGDG_EINVAL, "method must be PLAIN (0) or MATFREE (1)");
    }
    API_END
}

int sgdg_transform_1d_nnz(int k, int n, int which, int64_t* nnz) {
    API_BEGIN
    NEED(nnz);
    *nnz = transform_1d(k, n, which).nnz();
    API_END
}

int sgdg_transform_1d_export(int k, int n, int which, int64_t* rowptr, int32_t* col, double* val) {
    API_BEGIN
    NEED(rowptr);
    export_csr(transform_1d(k, n, which), rowptr, col, val);
    API_END
}

int sgdg_transform_nnz(int D, int k, int n, int scheme, int which, int64_t* nnz) {
    API_BEGIN
    NEED(nnz);
    *nnz = build_transform(D, k, n, scheme, which).nnz();
    API_END
}

int sgdg_transform_export(int D, int k, int n, int scheme, int which, int64_t* rowptr, int32_t* col, double* val) {
    API_BEGIN
    NEED(rowptr);
    export_csr(build_transform(D, k, n, scheme, which), rowptr, col, val);
    API_END
}

int sgdg_transform_device_export(int D, int k, int n, int scheme, int which, int64_t* nnz, int64_t* rowptr,
                                 int32_t* col, double* val) {
    API_BEGIN
    NEED(nnz);
    if (which < 0 || which > 3) throw Error(SGDG_EINVAL, "transform must be 0..3 (m2n, n2p, p2n, n2m)");
    if (k != 2 && k != 3 && k != 5) throw Error(SGDG_EINVAL, "the nodal basis exists for k = 2, 3, 5");
    require_gpu();
    const SparseIndex ix = make_index(D, k, n, scheme);
    cudaStream_t st = nullptr;
    CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    std::unique_ptr<DeviceCSR> A;
    try {
        A = gpu_transform(ix, transform_1d(k, n, which), st);
        const CSR h = download_csr(*A, st);
        *nnz = h.nnz();
        if (rowptr && col && val) export_csr(h, rowptr, col, val);
    } catch (...) {
        A.reset();
        cudaStreamDestroy(st);
        throw;
    }
    A.reset();
    cudaStreamDestroy(st);
    API_END
}

// ------------------------------------------------------------- Vlasov ----
int sgdg_vlasov_create(int D, int k, int n, int scheme, sgdg_vlasov** out) {
    API_BEGIN
    NEED(out);
    if (D < 1 || 2 * D > 8) throw Error(SGDG_EINVAL, "D (space dimensions) must be 1..4");
    if (k != 2 && k != 3 && k != 5) throw Error(SGDG_EINVAL, "the nodal basis exists for k = 2, 3, 5");
    auto v = std::make_unique<sgdg_vlasov>();
    v->D = D;
    v->P = 2 * D;
    v->k = k;
    v->n = n;
    v->ix = make_index(v->P, k, n, scheme);
    v->dlf = dlf1d(k, n);
    *out = v.release();
    API_END
}

int sgdg_vlasov_destroy(sgdg_vlasov* v) {
    API_BEGIN
    delete v;
    API_END
}

int sgdg_vlasov_size(const sgdg_vlasov* v, int64_t* N) {
    API_BEGIN
    NEED(v);
    NEED(N);
    *N = v->ix.N;
    API_END
}

int sgdg_vlasov_v_point(const sgdg_vlasov* v, double* out) {
    API_BEGIN
    NEED(v);
    NEED(out);
    if (!v->have_vpoint) {
        int ndev = 0;
        if (cudaGetDeviceCount(&ndev) == cudaSuccess && ndev > 0) {
            sgdg_vlasov* m = const_cast<sgdg_vlasov*>(v);
            Spare::Use use(*m);
            m->to_gpu();
        } else {
            cudaGetLastError();
            v->vpoint_host();
        }
    }
    std::copy(v->v_point.begin(), v->v_point.end(), out);
    API_END
}

int sgdg_vlasov_transform_nnz(const sgdg_vlasov* v, int which, int64_t* nnz) {
    API_BEGIN
    NEED(v);
    NEED(nnz);
    if (which < 0 || which > 3) throw Error(SGDG_EINVAL, "transform must be 0..3 (m2n, n2p, p2n, n2m)");
    *nnz = v->host_transform(which).nnz();
    API_END
}

int sgdg_vlasov_transform_export(const sgdg_vlasov* v, int which, int64_t* rowptr, int32_t* col, double* val) {
    API_BEGIN
    NEED(v);
    NEED(rowptr);
    if (which < 0 || which > 3) throw Error(SGDG_EINVAL, "transform must be 0..3 (m2n, n2p, p2n, n2m)");
    export_csr(v->host_transform(which), rowptr, col, val);
    API_END
}

int sgdg_vlasov_write_h5(const sgdg_vlasov* v, const char* path, int64_t nout, const double* times,
                         const double* states) {
    API_BEGIN
    NEED(v);
    NEED(path);
    if (nout < 0) throw Error(SGDG_EINVAL, "nout must be >= 0");
    if (nout > 0) {
        NEED(times);
        NEED(states);
    }
    H5Writer w(path);
    w.scalar_i64("dimensions", v->D);
    w.scalar_i64("order", v->k);
    w.scalar_i64("levels", v->n);
    static const char* names[4] = {"m2n", "n2p", "p2n", "n2m"};
    for (int t = 0; t < 4; t++) h5_write_csc(w, names[t], v->host_transform(t));
    for (int d = 0; d < v->P; d++)  // Ds[1] .. Ds[2D]: the 1-based names of the 0-based dimensions
        h5_write_csc(w, "Ds[" + std::to_string(d + 1) + "]", assemble_dd(v->ix, *v->dlf, d));
    if (nout > 0) {
        const int64_t N = v->ix.N;
        w.array_f64("times", times, nout);
        for (int64_t i = 0; i < nout; i++) {
            char name[32];
            std::snprintf(name, sizeof name, "f_modal.%06lld", (long long)(i + 1));
            w.array_f64(name, states + i * N, N);
        }
    }
    w.close();
    API_END
}

int sgdg_vlasov_rhs(sgdg_vlasov* v, const double* F_point, const double* f, double* out) {
    API_BEGIN
    NEED(v);
    NEED(F_point);
    NEED(f);
    NEED(out);
    const int64_t N = v->ix.N;
    const size_t b = sizeof(double) * (size_t)N;
    {
        Spare::Use use(*v);
        v->to_gpu();
    }
    DevBuf u(b), r(b);  // the sweeps may give way to them
    Spare::Use use(*v);
    CK(cudaMemcpyAsync(v->F.p, F_point, b * v->D, cudaMemcpyHostToDevice, v->stream));
    CK(cudaMemcpyAsync(u.p, f, b, cudaMemcpyHostToDevice, v->stream));
    int bad = 1;
    if (v->have_sweeps()) {
        CK(cudaMemsetAsync(v->flag.p, 0, sizeof(int), v->stream));
        CK(launch_check_finite(u.as<double>(), N, v->flag.as<int>(), v->stream));
        double* last = nullptr;
        CK(v->sweep_rhs(u.as<double>(), &last));
        CK(launch_sweep(v->last_sweep(), 1, last, r.as<double>(), v->flag.as<int>(), v->stream));
        CK(cudaMemcpyAsync(out, r.p, b, cudaMemcpyDeviceToHost, v->stream));
        CK(cudaMemcpyAsync(&bad, v->flag.p, sizeof(int), cudaMemcpyDeviceToHost, v->stream));
        CK(cudaStreamSynchronize(v->stream));
    }
    if (bad) {
        v->build_whole();
        CK(v->whole_rhs(u.as<double>()));
        CK(launch_csr_spmv(v->dT[3]->d, v->z.as<double>(), r.as<double>(), v->stream));
        CK(cudaMemcpyAsync(out, r.p, b, cudaMemcpyDeviceToHost, v->stream));
        CK(cudaStreamSynchronize(v->stream));
    }
    u.recycle();
    r.recycle();
    API_END
}

int sgdg_vlasov_evolve(sgdg_vlasov* v, const double* F_point, const double* f0, double t0, double t1, int64_t nsteps,
                       int nout, int method, double* times, double* states) {
    API_BEGIN
    NEED(v);
    NEED(F_point);
    NEED(f0);
    NEED(states);
    check_evolve_args(nsteps, nout, t0, t1);
    if (method == SGDG_METHOD_MATFREE) {
        if (!v->stream) {
            require_gpu();
            CK(cudaStreamCreateWithFlags(&v->stream, cudaStreamNonBlocking));
        }
        MFEngine eng(v->stream);
        SolveSpec sp{};
        sp.kind = MF_KIND_VLASOV;
        sp.D = v->P;
        sp.k = v->k;
        sp.n = v->n;
        sp.scheme = v->ix.scheme;
        sp.dt = (t1 - t0) / double(nsteps);
        sp.apply_dim = -1;
        const std::vector<float> w = vlasov_weights(v->ix, v->D, F_point);
        const int id = eng.add(sp, f0, w.data());
        auto steps = out_steps(nsteps, nout);
        int64_t done = 0;
        for (int i = 0; i < nout; i++) {
            eng.step(steps[i] - done);
            done = steps[i];
            eng.get_state(id, states + (size_t)i * v->ix.N);
            if (times) times[i] = t0 + (t1 - t0) * double(steps[i]) / double(nsteps);
        }
        eng.recycle();
        return SGDG_OK;
    }
    if (method != SGDG_METHOD_PLAIN) throw Error(SGDG_EINVAL, "method must be PLAIN (0) or MATFREE (1)");
    {
        Spare::Use use(*v);
        v->to_gpu();
    }
    cudaStream_t st = v->stream;
    const int64_t N = v->ix.N;
    const size_t b = sizeof(double) * (size_t)N;
    DevBuf y(b), acc(b), u0(b), u1(b);  // the sweeps may give way to them
    Spare::Use use(*v);
    CK(cudaMemcpyAsync(v->F.p, F_point, b * v->D, cudaMemcpyHostToDevice, st));
    const double dt = (t1 - t0) / double(nsteps);
    const double* in[4] = {y.as<double>(), u0.as<double>(), u1.as<double>(), u0.as<double>()};
    double* outv[4] = {u0.as<double>(), u1.as<double>(), u0.as<double>(), u1.as<double>()};
    int* flag = v->flag.as<int>();
    const auto steps = out_steps(nsteps, nout);
    // per stage the right-hand side in the nodal basis, then the last sweep (or
    // the whole) of n2m fused with the stage update; returns whether a stage
    // was not finite
    auto run = [&](bool whole) {
        StepGraph graph(1, nsteps >= kGraphStepsVlasov);
        auto launch = [&](int64_t n) {
            cudaError_t e = cudaSuccess;
            for (int64_t i = 0; i < n; i++)
                for (int stage = 1; stage <= 4 && e == cudaSuccess; stage++) {
                    double* last = v->z.as<double>();
                    e = whole ? v->whole_rhs(in[stage - 1]) : v->sweep_rhs(in[stage - 1], &last);
                    if (e == cudaSuccess)
                        e = whole ? launch_csr_rk4(v->dT[3]->d, last, y.as<double>(), acc.as<double>(), outv[stage - 1],
                                                   dt, stage, flag, st)
                                  : launch_csr_rk4(v->last_sweep(), last, y.as<double>(), acc.as<double>(),
                                                   outv[stage - 1], dt, stage, flag, st);
                }
            return e;
        };
        int bad = 0;
        int64_t done = 0;
        CK(cudaMemsetAsync(flag, 0, sizeof(int), st));
        CK(cudaMemcpyAsync(y.p, f0, b, cudaMemcpyHostToDevice, st));
        for (int i = 0; i < nout; i++) {
            graph.run(steps[i] - done, st, launch);
            done = steps[i];
            CK(cudaMemcpyAsync(states + (size_t)i * N, y.p, b, cudaMemcpyDeviceToHost, st));
            if (times) times[i] = t0 + (t1 - t0) * double(steps[i]) / double(nsteps);
        }
        CK(cudaMemcpyAsync(&bad, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        return bad != 0;
    };
    if (!v->have_sweeps() || run(false)) {
        v->build_whole();
        run(true);
    }
    for (DevBuf* w : {&y, &acc, &u0, &u1}) w->recycle();
    API_END
}

// ------------------------------------------------------------ batches ----
int sgdg_batch_create(sgdg_batch** out) {
    API_BEGIN
    NEED(out);
    require_gpu();
    auto b = std::make_unique<sgdg_batch>();
    CK(cudaStreamCreateWithFlags(&b->own, cudaStreamNonBlocking));
    b->eng.set_stream(b->own);
    *out = b.release();
    API_END
}

int sgdg_batch_destroy(sgdg_batch* b) {
    API_BEGIN
    delete b;  // cudaFree of the arenas waits for the batch's outstanding work
    API_END
}

int sgdg_batch_add(sgdg_batch* b, int kind, int D, int k, int n, int scheme, const double* a, double dt,
                   const double* y0, int* id) {
    API_BEGIN
    NEED(b);
    NEED(y0);
    NEED(id);
    if (kind != SGDG_KIND_ADVECT && kind != SGDG_KIND_WAVE) throw Error(SGDG_EINVAL, "kind must be ADVECT or WAVE");
    if (kind == SGDG_KIND_ADVECT) NEED(a);
    if (n < 2) throw Error(SGDG_EINVAL, "n must be >= 2");
    if (!std::isfinite(dt)) throw Error(SGDG_EINVAL, "dt must be finite");
    SolveSpec sp{};
    sp.kind = kind == SGDG_KIND_WAVE ? MF_KIND_WAVE : MF_KIND_ADVECT;
    sp.D = D;
    sp.k = k;
    sp.n = n;
    sp.scheme = scheme;
    for (int d = 0; d < D && d < 8; d++) sp.a[d] = a ? a[d] : 0.0;
    sp.dt = dt;
    sp.apply_dim = -1;
    *id = b->eng.add(sp, y0);
    API_END
}

int sgdg_batch_autotune(sgdg_batch* b, int* ntuned) {
    API_BEGIN
    NEED(b);
    const auto done = b->eng.autotune();
    if (ntuned) *ntuned = (int)done.size();
    API_END
}

int sgdg_tile_shape(int D, int k, int* wlog, int* coop, int* tuned) {
    API_BEGIN
    const MFTile t = mf_tile(D, k);
    if (wlog) *wlog = t.wlog;
    if (coop) *coop = t.coop;
    if (tuned) *tuned = mf_tile_tuned(D, k) ? 1 : 0;
    API_END
}

int sgdg_set_tile_shape(int D, int k, int wlog, int coop) {
    API_BEGIN
    if (D < 1 || D > 8 || k < 1 || k > 5) throw Error(SGDG_EINVAL, "tile shapes exist for 1 <= D <= 8, 1 <= k <= 5");
    mf_set_tile(D, k, MFTile{wlog, coop});
    API_END
}

int sgdg_clear_tile_shapes(void) {
    API_BEGIN
    mf_clear_tiles();
    API_END
}

int sgdg_batch_add_vlasov(sgdg_batch* b, int Dx, int k, int n, int scheme, double dt, const double* F_point,
                          const double* f0, int* id) {
    API_BEGIN
    NEED(b);
    NEED(F_point);
    NEED(f0);
    NEED(id);
    if (Dx < 1 || 2 * Dx > 8) throw Error(SGDG_EINVAL, "Dx (space dimensions) must be 1..4");
    if (!std::isfinite(dt)) throw Error(SGDG_EINVAL, "dt must be finite");
    SolveSpec sp{};
    sp.kind = MF_KIND_VLASOV;
    sp.D = 2 * Dx;
    sp.k = k;
    sp.n = n;
    sp.scheme = scheme;
    sp.dt = dt;
    sp.apply_dim = -1;
    const SparseIndex ix = make_index(sp.D, k, n, scheme);
    const std::vector<float> w = vlasov_weights(ix, Dx, F_point);
    *id = b->eng.add(sp, f0, w.data());
    API_END
}

int sgdg_batch_remove(sgdg_batch* b, int id) {
    API_BEGIN
    NEED(b);
    b->eng.remove(id);
    API_END
}

int sgdg_batch_set_stream(sgdg_batch* b, void* stream) {
    API_BEGIN
    NEED(b);
    b->eng.set_stream(stream ? (cudaStream_t)stream : b->own);
    API_END
}

int sgdg_batch_step(sgdg_batch* b, int64_t nsteps) {
    API_BEGIN
    NEED(b);
    if (nsteps < 0) throw Error(SGDG_EINVAL, "nsteps must be >= 0");
    b->eng.step(nsteps);
    API_END
}

int sgdg_batch_get_state(sgdg_batch* b, int id, double* y) {
    API_BEGIN
    NEED(b);
    NEED(y);
    b->eng.get_state(id, y);
    API_END
}

int sgdg_batch_state_size(sgdg_batch* b, int id, int64_t* len) {
    API_BEGIN
    NEED(b);
    NEED(len);
    *len = b->eng.state_size(id);
    API_END
}

int sgdg_batch_total_size(sgdg_batch* b, int64_t* len) {
    API_BEGIN
    NEED(b);
    NEED(len);
    *len = b->eng.total_size();
    API_END
}

int sgdg_batch_upload(sgdg_batch* b, const double* y_all) {
    API_BEGIN
    NEED(b);
    NEED(y_all);
    b->eng.upload_all(y_all);
    API_END
}

int sgdg_batch_download(sgdg_batch* b, double* y_all) {
    API_BEGIN
    NEED(b);
    NEED(y_all);
    b->eng.download_all(y_all);
    API_END
}

int sgdg_batch_step_host(sgdg_batch* b, const double* y_in, double* y_out, int64_t nsteps, int nchunks) {
    API_BEGIN
    NEED(b);
    NEED(y_in);
    NEED(y_out);
    b->eng.step_host(y_in, y_out, nsteps, nchunks);
    API_END
}

int sgdg_batch_step_info(sgdg_batch* b, int64_t* launches, double* dofs) {
    API_BEGIN
    NEED(b);
    if (launches) *launches = b->eng.launches_per_step();
    if (dofs) *dofs = b->eng.dof_updates_per_step();
    API_END
}

int sgdg_selftest_bounded_wait(double* seconds) {
    API_BEGIN
    require_gpu();
    cudaStream_t st = nullptr;
    CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    DevBuf buf(2 * sizeof(int));
    int err = 0;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaError_t e = cudaMemsetAsync(buf.p, 0, 2 * sizeof(int), st);
    if (e == cudaSuccess) e = cudaEventCreate(&e0);
    if (e == cudaSuccess) e = cudaEventCreate(&e1);
    if (e == cudaSuccess) e = cudaEventRecord(e0, st);
    // counter 0 must reach 1, and nothing ever increments it
    if (e == cudaSuccess) e = launch_wait_selftest(buf.as<int>(), 1, buf.as<int>() + 1, st);
    if (e == cudaSuccess) e = cudaEventRecord(e1, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&err, buf.as<int>() + 1, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaStreamDestroy(st);
    if (e != cudaSuccess) throw Error(SGDG_ECUDA, std::string("bounded wait self-test: ") + cudaGetErrorString(e));
    if (seconds) *seconds = ms / 1e3;
    if (!err) throw Error(SGDG_ECUDA, "bounded wait self-test: the wait did not report giving up");
    throw Error(SGDG_ETIMEOUT, "bounded wait gave up as designed");
    API_END
}

int sgdg_worklist_dryrun(int nclasses, const int* spec, int pass_only, int chunk, int nchunks, int64_t* items,
                         int64_t items_cap,
                         int64_t* nitems, int* nctr, int64_t* classes, int64_t* blockoff, int64_t boff_cap,
                         int64_t* nboff) {
    API_BEGIN
    NEED(spec);
    NEED(nitems);
    NEED(nboff);
    if (nclasses < 1 || nclasses > 4096) throw Error(SGDG_EINVAL, "nclasses must be in 1..4096");
    if (nchunks < 1 || nchunks > 64 || chunk < 0 || chunk >= nchunks)
        throw Error(SGDG_EINVAL, "chunk must be in 0..nchunks-1, nchunks in 1..64");
    struct Host {
        std::vector<std::vector<Pencil>> pencils;
        std::vector<int32_t> boff_index;
        std::vector<int64_t> boff;
    };
    std::vector<Host> host(nclasses);
    std::vector<WLClass> cls;
    for (int c = 0; c < nclasses; c++) {
        const int* q = spec + 8 * c;
        const int kind = q[0], D = q[1], k = q[2], n = q[3], scheme = q[4], ns = q[5], apply = q[6], adim = q[7];
        if (kind != MF_KIND_ADVECT && kind != MF_KIND_WAVE && kind != MF_KIND_VLASOV)
            throw Error(SGDG_EINVAL, "kind must be 0 (advection), 1 (wave) or 2 (Vlasov)");
        if (D < 1 || D > 8 || k < 1 || k > 5) throw Error(SGDG_EUNSUPPORTED, "matrix-free form supports D <= 8, k <= 5");
        if (ns < 1) throw Error(SGDG_EINVAL, "a class needs at least one solve");
        if (apply && (adim < -1 || adim >= D)) throw Error(SGDG_EINVAL, "apply dimension out of range");
        if (kind == MF_KIND_VLASOV && (apply || D % 2 != 0))
            throw Error(SGDG_EINVAL, "a Vlasov solve has an even phase-space dimension and steps");
        dlf1d(k, n);  // validates n
        const SparseIndex ix = make_index(D, k, n, scheme);
        Host& h = host[c];
        for (int d = 0; d < D; d++) {
            h.pencils.push_back(make_pencils(ix, d));
            for (auto& pc : h.pencils.back()) {
                h.boff_index.push_back((int32_t)h.boff.size());
                for (auto o : pc.blockoff) h.boff.push_back(o);
            }
        }
        const int64_t Ns = kind == MF_KIND_WAVE && !apply ? 2 * ix.N : ix.N;
        if ((int64_t)ns * Ns >= (int64_t(1) << 31))
            throw Error(SGDG_EUNSUPPORTED, "a class of solves holds more than 2^31 coefficients");
        cls.push_back(WLClass{kind, D, k, n, apply != 0, apply ? adim : -1, ix.N, Ns, ns, h.pencils, h.boff_index});
    }
    std::vector<MFItem> list;
    int nc = 0;
    mf_work_list(cls, list, nc, pass_only != 0, nullptr, chunk, nchunks, nullptr);
    int64_t nb = 0;
    for (auto& h : host) nb += (int64_t)h.boff.size();
    *nitems = (int64_t)list.size();
    *nboff = nb;
    if (nctr) *nctr = nc;
    if (items && items_cap >= (int64_t)list.size()) {
        for (size_t i = 0; i < list.size(); i++) {
            const MFItem& it = list[i];
            const int64_t f[SGDG_WL_FIELDS] = {it.cls,      it.d,        it.tab,      it.flags,    it.src,
                                               it.dst,      it.wsel,     it.stage,    it.wait_ctr, it.wait_need,
                                               it.win_ctr,  it.win_need, it.done_ctr, it.lmax,     it.lp,
                                               it.boff,     it.R,        it.g0,       it.W,        it.Wv,
                                               it.kd1,      it.kDm1,     it.rlong,    it.rmagic,   it.rshift};
            std::copy(f, f + SGDG_WL_FIELDS, items + i * SGDG_WL_FIELDS);
        }
    }
    if (classes) {
        int64_t first = 0;
        for (int c = 0; c < nclasses; c++) {
            classes[4 * c] = cls[c].N;
            classes[4 * c + 1] = cls[c].Ns;
            classes[4 * c + 2] = cls[c].nslots;
            classes[4 * c + 3] = first;
            first += (int64_t)host[c].boff.size();
        }
    }
    if (blockoff && boff_cap >= nb) {
        int64_t o = 0;
        for (auto& h : host) {
            std::copy(h.boff.begin(), h.boff.end(), blockoff + o);
            o += (int64_t)h.boff.size();
        }
    }
    API_END
}

int sgdg_selftest_convert(const double* x, int64_t n, int64_t* mismatches, int64_t* first) {
    API_BEGIN
    require_gpu();
    if (n < 0) throw Error(SGDG_EINVAL, "n must be >= 0");
    if (n > 0) NEED(x);
    cudaStream_t st = nullptr;
    CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    DevBuf xs((size_t)(n > 0 ? n : 1) * sizeof(double));
    DevBuf bad(2 * sizeof(unsigned long long));
    unsigned long long out[2] = {0ull, ~0ull};
    cudaError_t e = cudaMemcpyAsync(bad.p, out, sizeof(out), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && n > 0) e = cudaMemcpyAsync(xs.p, x, (size_t)n * sizeof(double), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = launch_convert_selftest(xs.as<double>(), n, bad.as<unsigned long long>(), st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, bad.p, sizeof(out), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    if (e != cudaSuccess) throw Error(SGDG_ECUDA, std::string("conversion self-test: ") + cudaGetErrorString(e));
    if (mismatches) *mismatches = (int64_t)out[0];
    if (first) *first = out[0] ? (int64_t)out[1] : -1;
    API_END
}

int sgdg_set_hbm_budget(int64_t bytes) {
    API_BEGIN
    if (bytes < 0) throw Error(SGDG_EINVAL, "budget must be >= 0");
    g_budget = bytes;
    g_budget_set++;
    device_pool().trim(bytes > 0 ? (size_t)std::max<int64_t>(0, bytes - g_in_use.load()) : 0);
    API_END
}

int sgdg_hbm_in_use(int64_t* bytes) {
    API_BEGIN
    NEED(bytes);
    *bytes = g_in_use.load();
    API_END
}

int sgdg_sync(void) {
    API_BEGIN
    require_gpu();
    CK(cudaDeviceSynchronize());
    API_END
}

}  // extern "C"

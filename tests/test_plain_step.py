"""Stepping of the plain form: operators without the entries that hold only
the rounding of a zero, several solves per row, short and long rows."""
import numpy as np
import pytest


def rk4(A, y, dt, nsteps):
    for _ in range(nsteps):
        k1 = A @ y
        k2 = A @ (y + 0.5 * dt * k1)
        k3 = A @ (y + 0.5 * dt * k2)
        y = y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + A @ (y + dt * k3))
    return y


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("n", [2, 4, 6])
def test_rounding_of_zeros_is_far_below_the_other_entries(sgdg, k, n):
    # the bound 1e-10 lies in a gap of the 1D operator and of the squares of
    # its leading blocks: at least a factor of 5 above what is dropped and
    # 1e5 below what is kept (rounding at k = 5 reaches 2e-12 and 1e-11)
    A = sgdg.periodic_DLF_matrix(k, n).toarray()
    rel = np.abs(A) / np.abs(A).max()
    assert not np.any((rel > 2e-11) & (rel < 1e-5))
    B = np.where(rel > 1e-10, A, 0.0)
    for levels in range(1, n + 2):
        b = B[:k << (levels - 1), :k << (levels - 1)]
        sums, terms = np.abs(b @ b), np.abs(b) @ np.abs(b)
        rel2 = sums[terms > 0] / terms[terms > 0]
        assert not np.any((rel2 > 2e-11) & (rel2 < 1e-5))


SHAPES = [(1, 1, 2, "sparse"), (1, 5, 8, "sparse"), (2, 1, 4, "sparse"), (2, 4, 3, "full"), (3, 3, 4, "sparse"),
          (2, 6, 3, "sparse"), (1, 8, 7, "sparse"), (4, 2, 3, "sparse")]


@pytest.mark.gpu
@pytest.mark.parametrize("D,k,n,scheme", SHAPES)
def test_evolvers_against_the_whole_operator(sgdg, D, k, n, scheme):
    # launched as they are, and as 8-step graphs and what is left over of them; per step
    # a result is off by a few roundings of dt |A| |y|, plus the dropped
    # entries (2e-12 of the largest): 1e-10 of the state covers 259 steps at
    # dt |A| <= 1/8
    op = sgdg.SparseGridOperator(D, k, n, scheme)
    rng = np.random.default_rng(D * 100 + k * 10 + n)
    N = op.N
    a = rng.uniform(-1, 1, D)
    G = sum(-a[d] * op.csr(d + 1) for d in range(D))
    W = op.csr(-1)
    for A, y, evolve in ((W, rng.standard_normal(2 * N), "wave"), (G, rng.standard_normal(N), "advect")):
        dt = 1.0 / max(np.abs(A).sum(1).max(), 1e-3) if evolve == "advect" else \
            1.0 / np.sqrt(max(np.abs(A).sum(1).max(), 1e-3))
        for steps, h in ((1, dt), (7, dt), (17, dt), (259, dt / 8)):
            ref = rk4(A, y, h, steps)
            if evolve == "wave":
                _, st = sgdg.wave_evolve(D, k, n, y[:N], y[N:], 0.0, steps * h, nsteps=steps, scheme=scheme, op=op)
            else:
                _, st = sgdg.advect_evolve(D, k, n, a, y, 0.0, steps * h, nsteps=steps, scheme=scheme, op=op)
            assert np.linalg.norm(st[-1] - ref) <= 1e-10 * np.linalg.norm(ref), (evolve, steps)


@pytest.mark.gpu
@pytest.mark.parametrize("D,k,n", [(2, 3, 4), (1, 8, 9)])
@pytest.mark.parametrize("solves", [1, 2, 3, 4, 5, 18])
def test_solves_of_a_set_equal_their_own_evolution(sgdg, D, k, n, solves):
    # sets of 1, 2 and 4 with a remainder, and (1D k=8 n=9, rows of 4096
    # entries) rows in segments; bit for bit
    import torch
    op = sgdg.SparseGridOperator(D, k, n)
    N, dt, steps = op.N, 1e-6, 3
    y = np.random.default_rng(solves).standard_normal((solves, 2 * N))
    dev = torch.tensor(y, device="cuda")
    op.plain_steps_device(dev.data_ptr(), solves, dt, steps)
    got = dev.cpu().numpy()
    for i in range(solves):
        t1 = steps * dt
        _, st = sgdg.wave_evolve(D, k, n, y[i, :N], y[i, N:], 0.0, t1, nsteps=steps, op=op)
        assert t1 / steps != dt or np.array_equal(got[i], st[-1]), i
        assert np.allclose(got[i], st[-1], rtol=0, atol=1e-12 * np.abs(st[-1]).max())


@pytest.mark.gpu
@pytest.mark.parametrize("where,value", [(0, np.nan), (-1, np.inf), (7, -np.inf), (None, 1e306)])
def test_what_is_not_finite_spreads_as_the_whole_operator_spreads_it(sgdg, where, value):
    import torch
    D, k, n, dt = 2, 3, 4, 1e-2
    op = sgdg.SparseGridOperator(D, k, n)
    N = op.N
    rng = np.random.default_rng(3)
    y = rng.standard_normal(2 * N)
    if where is None:
        y *= value
    else:
        y[where] = value
    a = rng.uniform(-1, 1, D)
    G = sum(-a[d] * op.csr(d + 1) for d in range(D))
    fine = rng.standard_normal(2 * N)
    with np.errstate(all="ignore"):
        ref = rk4(op.csr(-1), y, dt, 2)
        ref_a = rk4(G, y[:N], dt, 1)
    _, st = sgdg.wave_evolve(D, k, n, y[:N], y[N:], 0.0, 2 * dt, nsteps=2, op=op)
    assert np.array_equal(np.isfinite(st[-1]), np.isfinite(ref))
    _, st = sgdg.advect_evolve(D, k, n, a, y[:N], 0.0, dt, nsteps=1, op=op)
    assert np.array_equal(np.isfinite(st[-1]), np.isfinite(ref_a))
    dev = torch.tensor(np.concatenate([y, fine]), device="cuda")
    op.plain_steps_device(dev.data_ptr(), 2, dt, 2)
    got = dev.cpu().numpy().reshape(2, -1)
    assert np.array_equal(np.isfinite(got[0]), np.isfinite(ref)) and np.all(np.isfinite(got[1]))


@pytest.mark.gpu
def test_stepping_at_a_memory_limit(sgdg):
    # no room to keep the states of the call's start, or for sets padded to
    # whole ones: the whole operator steps them one by one in three scratch
    # vectors; a budget below those is refused
    import torch
    D, k, n, solves, dt = 2, 3, 5, 65, 1e-4
    op = sgdg.SparseGridOperator(D, k, n)
    N = op.N
    y = torch.tensor(np.random.default_rng(0).standard_normal(solves * 2 * N), device="cuda")
    one, two, three = y.clone(), y.clone(), y.clone()
    op.plain_steps_device(one.data_ptr(), solves, dt, 2)
    op.device_csr(-1)  # the whole operator is there before the limit
    try:
        sgdg.set_hbm_budget(sgdg.hbm_in_use() + 8 * solves * 2 * N * 3 + 64)
        op.plain_steps_device(two.data_ptr(), solves, dt, 2)
        assert float((one - two).norm() / one.norm()) < 1e-12
        sgdg.set_hbm_budget(sgdg.hbm_in_use() + 8 * solves * 2 * N * 2)
        with pytest.raises(sgdg.SGDGError) as e:
            op.plain_steps_device(three.data_ptr(), solves, dt, 2)
        assert e.value.code == 2 and torch.equal(three, y)
    finally:
        sgdg.set_hbm_budget(0)


@pytest.mark.gpu
@pytest.mark.parametrize("D,k,n,which", [(4, 2, 6, 0), (2, 3, 7, 0), (1, 3, 10, 0), (3, 3, 6, -1)])
def test_application_with_the_pruned_operator(sgdg, D, k, n, which):
    # either side of the size from which applications go through the pruned
    # operator (4D: just above, 2D: just below; 1D: rows of 3072 entries).  The
    # entries dropped are 2e-12 of the largest and the sums as long as a line:
    # 1e-10 of the result for random vectors, whose result the largest entries make
    op = sgdg.SparseGridOperator(D, k, n)
    A = op.csr(which)
    x = np.random.default_rng(D).standard_normal(A.shape[0])
    ref = A @ x
    assert np.linalg.norm(op.apply(x, which) - ref) <= 1e-10 * np.linalg.norm(ref)
    for where, value in ((0, np.nan), (A.shape[0] - 1, np.inf), (A.shape[0] // 3, -np.inf)):
        z = x.copy()
        z[where] = value
        with np.errstate(all="ignore"):
            bad = A @ z
        y = op.apply(z, which)
        assert np.array_equal(np.isfinite(y), np.isfinite(bad)) and np.array_equal(np.isnan(y), np.isnan(bad))
        fin = np.isfinite(bad)
        assert np.linalg.norm(y[fin] - bad[fin]) <= 1e-10 * np.linalg.norm(ref)
    assert np.linalg.norm(op.apply(x, which) - ref) <= 1e-10 * np.linalg.norm(ref)  # and finite data again


@pytest.mark.gpu
def test_applications_in_a_graph_and_on_two_streams(sgdg):
    import torch
    op = sgdg.SparseGridOperator(4, 2, 6)
    A = op.csr(0)
    x = torch.tensor(np.random.default_rng(1).standard_normal((2, op.N)), device="cuda")
    y = torch.zeros_like(x)
    op.apply_device(x[0].data_ptr(), y[0].data_ptr(), which=0)  # assembles
    torch.cuda.synchronize()
    ref = np.stack([A @ v for v in x.cpu().numpy()])
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for i in range(40):
        op.apply_device(x[i % 2].data_ptr(), y[i % 2].data_ptr(), which=0, stream=streams[i % 2].cuda_stream)
    torch.cuda.synchronize()
    assert np.linalg.norm(y.cpu().numpy() - ref) <= 1e-10 * np.linalg.norm(ref)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        op.apply_device(x[0].data_ptr(), y[0].data_ptr(), which=0, stream=streams[0].cuda_stream)
    for value in (1.0, float("nan"), 2.0):
        x[0, 5] = value
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        with np.errstate(all="ignore"):
            ref = A @ x[0].cpu().numpy()
        got = y[0].cpu().numpy()
        fin = np.isfinite(ref)
        assert np.array_equal(np.isfinite(got), fin)
        assert np.linalg.norm(got[fin] - ref[fin]) <= 1e-10 * np.linalg.norm(ref[fin])


@pytest.mark.gpu
@pytest.mark.parametrize("k,n", [(2, 5), (3, 5)])
def test_stepping_against_the_operator_in_plain_numpy(sgdg, k, n):
    # both operators are within 1e-14 of their largest entry of the true one
    # (numpy's: rounding of Q' A Q, 4e-15 at k=3 n=5; the wavelets' own, in both,
    # 2e-15 there, but 2e-13 at k=4 and 8e-13 at k=5; the reference's route is
    # 6e-14 to 4e-13 away), and what that changes in a step is at most its
    # share of dt |L| <= 3, with a factor 2 for the norms: 6e-14 in each of 30 steps
    import importlib.util
    import pathlib
    path = pathlib.Path(__file__).resolve().parents[1] / "perf" / "cases.py"
    spec = importlib.util.spec_from_file_location("perf_cases", path)
    cases = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(cases)
    D, _ = cases.derivative_1d(k, n)
    N = len(D)
    A = np.block([[np.zeros((N, N)), np.eye(N)], [D @ D, np.zeros((N, N))]])
    rng = np.random.default_rng(k)
    y = rng.standard_normal(2 * N)
    y[N:] *= np.linalg.norm(D, 2)  # velocities of the size the fastest modes have
    dt = 1.0 / np.linalg.norm(D, 2)
    _, st = sgdg.wave_evolve(1, k, n, y[:N], y[N:], 0.0, 30 * dt, nsteps=30)
    ref = rk4(A, y, dt, 30)
    got = np.asarray(st[-1]).reshape(-1)
    assert np.linalg.norm(got[:N] - ref[:N]) <= 30 * 6e-14 * np.linalg.norm(ref[:N])


@pytest.mark.gpu
@pytest.mark.parametrize("D,k,n", [(2, 3, 8), (2, 3, 9), (2, 4, 7), (2, 4, 8)])
def test_finest_grids_step_with_the_whole_operator(sgdg, D, k, n):
    # k + n on both sides of the limit of the pruned wave operator: the states are
    # of the size of the largest entries' results, of which the two operators
    # differ by at most 1e-11 per step, and with the whole one by roundings
    op = sgdg.SparseGridOperator(D, k, n)
    A, N = op.csr(-1), op.N
    y = np.random.default_rng(n).standard_normal(2 * N)
    dt = 1.0 / np.sqrt(np.abs(A).sum(1).max())
    _, st = sgdg.wave_evolve(D, k, n, y[:N], y[N:], 0.0, 3 * dt, nsteps=3, op=op)
    ref = rk4(A, y, dt, 3)
    assert np.linalg.norm(st[-1] - ref) <= (1e-10 if k + n <= 11 else 1e-13) * np.linalg.norm(ref)

"""Calls at a memory limit that holds the whole operators and the call's own
vectors: they go without the pruned ones, and a handle that holds one gives it
back where another call needs the room."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def budget(sgdg):
    def room(extra):  # device bytes beside what is in use now
        sgdg.set_hbm_budget(sgdg.hbm_in_use() + extra)
    yield room
    sgdg.set_hbm_budget(0)


@pytest.mark.parametrize("host", [False, True])
def test_application_without_room_for_the_pruned_operator(sgdg, budget, host):
    import torch
    op = sgdg.SparseGridOperator(4, 2, 6)  # 1.6 M entries: applied pruned where there is room
    op.device_csr(0)
    x = np.random.default_rng(0).standard_normal(op.N)
    ref = op.csr(0) @ x
    budget(2 * 8 * op.N + 64 if host else 64)
    for _ in range(2):
        if host:
            y = op.apply(x, 0)
        else:
            xd = torch.tensor(x, device="cuda")
            yd = torch.zeros_like(xd)
            op.apply_device(xd.data_ptr(), yd.data_ptr(), which=0)
            torch.cuda.synchronize()
            y = yd.cpu().numpy()
        # sums of at most 2000 terms, either operator (their entries differ by 2e-12 of the largest)
        assert np.linalg.norm(y - ref) <= 1e-10 * np.linalg.norm(ref)
    op.close()


def test_application_gives_the_pruned_operator_back(sgdg, budget):
    big = sgdg.SparseGridOperator(4, 2, 6)
    x = np.random.default_rng(1).standard_normal(big.N)
    big.device_csr(0)
    whole = sgdg.hbm_in_use()
    first = big.apply(x, 0)
    assert sgdg.hbm_in_use() > whole + (1 << 20)
    small = sgdg.SparseGridOperator(2, 3, 4)
    budget(2 * 8 * big.N + 64)  # the vectors of the application, not another operator
    assert np.array_equal(big.apply(x, 0), first)
    y = np.random.default_rng(2).standard_normal(small.N)
    budget(0)
    assert np.allclose(small.apply(y, 0), small.csr(0) @ y, rtol=0, atol=1e-9 * np.abs(small.csr(0)).max())
    # and goes on with the whole one
    sgdg.set_hbm_budget(sgdg.hbm_in_use() + 2 * 8 * big.N + 64)
    assert np.linalg.norm(big.apply(x, 0) - first) <= 1e-10 * np.linalg.norm(first)
    big.close()
    small.close()


def rk4(A, y, dt, nsteps):
    for _ in range(nsteps):
        k1 = A @ y
        k2 = A @ (y + 0.5 * dt * k1)
        k3 = A @ (y + 0.5 * dt * k2)
        y = y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + A @ (y + dt * k3))
    return y


def wave(sgdg, op, y, dt=1e-4, steps=3):
    _, st = sgdg.wave_evolve(op.D, op.k, op.n, y[:op.N], y[op.N:], 0.0, steps * dt, nsteps=steps, op=op)
    return st[-1]


def advect(sgdg, op, y, dt=1e-4, steps=3):
    a = np.linspace(0.5, 1.0, op.D)
    _, st = sgdg.advect_evolve(op.D, op.k, op.n, a, y[:op.N], 0.0, steps * dt, nsteps=steps, op=op)
    return st[-1]


def vectors(op):  # of a wave's evolution
    return 4 * 8 * 2 * op.N + 64


def test_wave_without_room_for_the_pruned_operator(sgdg, budget):
    # the whole operator is there, or a run that was not finite has built it
    op = sgdg.SparseGridOperator(3, 3, 5)
    y = np.random.default_rng(0).standard_normal(2 * op.N)
    ref = rk4(op.csr(-1), y, 1e-4, 3)
    op.device_csr(-1)
    budget(vectors(op))
    for _ in range(2):
        assert np.linalg.norm(wave(sgdg, op, y) - ref) <= 1e-10 * np.linalg.norm(ref)
    sgdg.set_hbm_budget(0)
    got = wave(sgdg, op, y)  # with the pruned one again
    bad = y.copy()
    bad[3] = np.nan
    assert not np.all(np.isfinite(wave(sgdg, op, bad)))
    budget(0)  # the pruned one makes room for the vectors
    assert np.linalg.norm(wave(sgdg, op, y) - got) <= 1e-10 * np.linalg.norm(got)
    op.close()


def test_advection_gives_its_operator_back(sgdg, budget):
    op, other = sgdg.SparseGridOperator(3, 3, 6), sgdg.SparseGridOperator(3, 2, 4)
    y = np.random.default_rng(1).standard_normal(op.N)
    before = sgdg.hbm_in_use()
    first = advect(sgdg, op, y)
    assert sgdg.hbm_in_use() > before + (1 << 20)  # kept for the next call
    budget(0)
    z = np.random.default_rng(2).standard_normal(2 * other.N)
    ref = rk4(other.csr(-1), z, 1e-4, 3)
    assert np.linalg.norm(wave(sgdg, other, z) - ref) <= 1e-10 * np.linalg.norm(ref)
    # and back again, whichever operator fits now
    sgdg.set_hbm_budget(0)
    assert np.array_equal(advect(sgdg, op, y), first)
    op.close()
    other.close()


@pytest.mark.parametrize("evolve", [wave, advect])
def test_a_run_after_one_that_was_not_finite(sgdg, budget, evolve):
    # at every budget under which a run that is not finite fits, on a fresh handle
    # as in a sequence, a finite one does as well
    y = np.random.default_rng(3).standard_normal(2 * sgdg.get_size(3, 3, 5))
    bad = y.copy()
    bad[3] = np.inf
    ran = 0
    for extra in np.geomspace(1 << 20, 64 << 20, 13):
        op = sgdg.SparseGridOperator(3, 3, 5)
        budget(int(extra))
        try:
            evolve(sgdg, op, bad)
        except sgdg.SGDGError as e:
            assert e.code == 2
        else:
            ran += 1
            assert np.all(np.isfinite(evolve(sgdg, op, y)))
            assert not np.all(np.isfinite(evolve(sgdg, op, bad)))
            assert np.all(np.isfinite(evolve(sgdg, op, y)))
        sgdg.set_hbm_budget(0)
        op.close()
    assert 0 < ran < 13


def vlasov(sgdg, seed=5):
    v = sgdg.VlasovOperator(2, 2, 4)
    rng = np.random.default_rng(seed)
    return v, rng.standard_normal((2, v.N)), rng.standard_normal(v.N)


def test_vlasov_without_room_for_the_sweeps(sgdg, budget):
    v, F, f = vlasov(sgdg)
    ref = v.rhs(F, f)
    bad = f.copy()
    bad[3] = np.nan
    assert not np.all(np.isfinite(v.rhs(F, bad)))  # builds the assembled operators

    def evolve():
        return sgdg.vlasov_evolve(2, 2, 4, F, f, 0.0, 3e-4, nsteps=3, op=v)[1][-1]
    evolved = evolve()
    for call in range(2):
        budget(0)  # the sweeps make room for the vectors
        got = evolve() if call else v.rhs(F, f)
        want = evolved if call else ref
        # the same right-hand side in another order of its sums (at most 1e4 terms of the
        # size of the largest, which a transform grows by less than 100)
        assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want)
        sgdg.set_hbm_budget(0)
        assert np.array_equal(v.rhs(F, f), ref)  # with the sweeps again
    v.close()


def test_vlasov_run_after_one_that_was_not_finite(sgdg, budget):
    ran = 0
    for extra in np.geomspace(1 << 18, 256 << 20, 21):
        v, F, f = vlasov(sgdg)
        bad = f.copy()
        bad[3] = np.inf
        budget(int(extra))
        try:
            v.rhs(F, bad)
        except sgdg.SGDGError as e:
            assert e.code == 2
        else:
            ran += 1
            assert np.all(np.isfinite(v.rhs(F, f)))
            assert not np.all(np.isfinite(v.rhs(F, bad)))
            assert np.all(np.isfinite(v.rhs(F, f)))
        sgdg.set_hbm_budget(0)
        v.close()
    assert 0 < ran < 21


def test_many_points_without_room_for_the_pencils(sgdg, budget):
    D, k, n, points = 3, 4, 3, 1 << 15
    rng = np.random.default_rng(7)
    c = rng.standard_normal(sgdg.get_size(D, k, n))
    x = rng.uniform(0, 1, (points, D))
    few = [sgdg.reconstruct_DG(D, k, n, c, part) for part in np.array_split(x, 16)]  # block by block
    budget(8 * (c.size + points * (D + 1)) + 64)
    for _ in range(2):
        assert np.array_equal(sgdg.reconstruct_DG(D, k, n, c, x), np.concatenate(few))
    sgdg.set_hbm_budget(0)
    # the sums in another order: 1e3 terms a point at most, none above |c| 8^1.5 k^1.5 = 500
    assert np.allclose(sgdg.reconstruct_DG(D, k, n, c, x), np.concatenate(few), rtol=0, atol=1e-10)

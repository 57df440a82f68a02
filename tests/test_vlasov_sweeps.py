"""The plain Vlasov right-hand side as sweeps along the dimensions, against the
assembled transforms and derivatives it replaces."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def assembled(sgdg, D, k, n, scheme, F, v):
    """The right-hand side from the assembled operators (src/pdes.jl:174-192)."""
    P = 2 * D
    T = [sgdg.transform(P, k, n, *w, scheme=scheme) for w in
         (("modal", "nodal"), ("nodal", "points"), ("points", "nodal"), ("nodal", "modal"))]
    Ds = sgdg.grad_matrix(P, k, n, scheme)

    def rhs(f):
        pt = [T[1] @ (T[0] @ (A @ f)) for A in Ds]
        c = -sum(v[d] * pt[d] for d in range(D)) + sum(F[d] * pt[D + d] for d in range(D))
        return T[3] @ (T[2] @ c)
    return rhs


# P = 2, 4 and 8 (4 vectors at a time), 6 (2 at a time); lines of 2 to 640 elements;
# transforms in pairs of dimensions and (1x1v n=7, 2x2v n=6 and k=3 n=5) one by one
CASES = [(1, 2, 2, "sparse"), (1, 5, 7, "sparse"), (1, 3, 4, "full"), (2, 2, 4, "sparse"), (2, 3, 3, "sparse"),
         (2, 5, 2, "sparse"), (3, 2, 2, "sparse"), (4, 2, 2, "sparse"),
         (2, 2, 6, "sparse"), (2, 3, 5, "sparse")]


@pytest.mark.parametrize("D,k,n,scheme", CASES)
def test_right_hand_side_and_steps(sgdg, D, k, n, scheme):
    # a transform's entries are at most a few units and its products below
    # 1e-12 are dropped by the assembled one only: 1e-10 of the result covers
    # the sums of a row (at most 1e2 of its terms' size at these shapes)
    op = sgdg.VlasovOperator(D, k, n, scheme)
    rng = np.random.default_rng(10 * D + k)
    N = op.N
    F, f = rng.uniform(-1, 1, (D, N)), rng.standard_normal(N)
    rhs = assembled(sgdg, D, k, n, scheme, F, op.v_point())
    ref = rhs(f)
    assert np.linalg.norm(op.rhs(F, f) - ref) <= 1e-10 * np.linalg.norm(ref)
    dt = 0.1 * np.linalg.norm(f) / np.linalg.norm(ref)
    for steps in (1, 17):  # launched one by one, and as a graph
        y = f
        for _ in range(steps):
            k1 = rhs(y)
            k2 = rhs(y + 0.5 * dt * k1)
            k3 = rhs(y + 0.5 * dt * k2)
            y = y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + rhs(y + dt * k3))
        _, st = sgdg.vlasov_evolve(D, k, n, F, f, 0.0, steps * dt, nsteps=steps, op=op, scheme=scheme)
        assert np.linalg.norm(st[-1] - y) <= 1e-9 * np.linalg.norm(y), steps
    op.close()


# grids whose launches are all resident (ascending rows), partly (the derivatives
# are more blocks than the sweeps) and all larger (long rows first)
@pytest.mark.parametrize("D,k,n,scheme", [(2, 2, 5, "sparse"), (2, 2, 7, "sparse"), (1, 2, 7, "full"), (1, 3, 7, "full")])
def test_right_hand_side_of_small_and_large_launches(sgdg, D, k, n, scheme):
    # as above: 1e-10 of the result
    op = sgdg.VlasovOperator(D, k, n, scheme)
    rng = np.random.default_rng(D + n)
    F, f = rng.uniform(-1, 1, (D, op.N)), rng.standard_normal(op.N)
    ref = assembled(sgdg, D, k, n, scheme, F, op.v_point())(f)
    assert np.linalg.norm(op.rhs(F, f) - ref) <= 1e-10 * np.linalg.norm(ref)
    op.close()


@pytest.mark.parametrize("where,value", [(0, np.nan), (3, np.inf), (-1, -np.inf)])
def test_what_is_not_finite_spreads_as_the_assembled_operators_spread_it(sgdg, where, value):
    D, k, n = 1, 3, 4
    op = sgdg.VlasovOperator(D, k, n)
    rng = np.random.default_rng(5)
    F, f = rng.uniform(-1, 1, (D, op.N)), rng.standard_normal(op.N)
    rhs = assembled(sgdg, D, k, n, "sparse", F, op.v_point())
    f[where] = value
    with np.errstate(all="ignore"):
        ref = rhs(f)
        y = f + 1e-3 * ref  # the pattern of one step contains that of its first stage
    assert np.array_equal(np.isfinite(op.rhs(F, f)), np.isfinite(ref))
    _, st = sgdg.vlasov_evolve(D, k, n, F, f, 0.0, 1e-3, nsteps=1, op=op)
    assert not np.any(np.isfinite(st[-1]) & ~np.isfinite(y))
    f[where] = 0.0  # and the handle goes on with finite data
    ref = rhs(f)
    assert np.linalg.norm(op.rhs(F, f) - ref) <= 1e-10 * np.linalg.norm(ref)
    op.close()


def test_one_handle_for_both_forms(sgdg):
    W = importlib.import_module(sgdg.__name__ + ".workloads")
    F, f0 = W.vlasov_case(sgdg, 1, 2, 4, seed=5)
    op = sgdg.VlasovOperator(1, 2, 4)
    _, mf = sgdg.vlasov_evolve(1, 2, 4, F, f0, 0.0, 5e-3, nsteps=5, op=op, method="matfree")
    _, pl = sgdg.vlasov_evolve(1, 2, 4, F, f0, 0.0, 5e-3, nsteps=5, op=op)
    assert np.linalg.norm(mf[-1] - pl[-1]) <= 1e-6 * np.linalg.norm(pl[-1])
    op.close()

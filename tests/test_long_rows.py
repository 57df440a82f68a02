"""Steps with rows of more than 2,048 entries, which are summed in segments: few of
them, all resident at once, and more, with last segments of one to 2,047 entries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# segments: 54 (remainders of 254 to 1,023), 4,560 and 32,736 (of 1 to 38), 5,120 (of 512), 8,192 (none)
@pytest.mark.parametrize("D,k,n", [(2, 3, 9), (2, 2, 10), (2, 4, 9), (1, 5, 9), (1, 8, 9)])
def test_steps_with_long_rows(sgdg, D, k, n):
    op = sgdg.SparseGridOperator(D, k, n)
    A = op.csr(-1)
    W = abs(A)
    longest = int(np.diff(A.indptr).max())
    assert longest > 2048
    y = np.random.default_rng(0).standard_normal(2 * op.N)
    y[np.random.default_rng(1).integers(0, 2 * op.N, op.N)] *= 1e3
    dt = 0.5 / np.sqrt(np.asarray(W[op.N:].sum(axis=1)).max())

    k1 = A @ y
    k2 = A @ (y + 0.5 * dt * k1)
    k3 = A @ (y + 0.5 * dt * k2)
    want = y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + A @ (y + dt * k3))
    _, got = sgdg.wave_evolve(D, k, n, y[:op.N], y[op.N:], 0.0, dt, nsteps=1, op=op)
    # Either side rounds each sum to `longest` units of the sum of its magnitudes, the
    # errors of four stages travel on: sum_j (dt W)^j |y| / j! bounds both.  The device's
    # operator holds the same entries as the host's.
    size, term = np.abs(y), np.abs(y)
    for j in range(1, 5):
        term = dt / j * (W @ term)
        size = size + term
    eps = np.finfo(float).eps
    assert np.all(np.abs(got[-1] - want) <= 4 * (longest + 8) * eps * size)
    op.close()

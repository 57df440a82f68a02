"""Point evaluation at many points (levels summed along dimension 1 once for
all of them) against the block-by-block evaluation of fewer points and the
oracle."""
import numpy as np
import pytest

from test_evaluate import edge_points

pytestmark = pytest.mark.gpu

# blocks of 1 to 125 numbers padded to 4; one and several outer modes; lines of one level
CASES = [(1, 1, 9, "sparse"), (1, 5, 6, "sparse"), (2, 2, 6, "sparse"), (2, 3, 4, "full"), (2, 5, 5, "sparse"),
         (3, 1, 5, "sparse"), (3, 2, 5, "sparse"), (3, 3, 4, "sparse"), (3, 4, 3, "full"), (3, 5, 3, "sparse"),
         (4, 3, 3, "sparse"), (5, 2, 2, "sparse"), (2, 3, 1, "sparse"), (3, 3, 0, "sparse")]


def in_parts(sgdg, D, k, n, c, pts, scheme):
    return np.concatenate([sgdg.reconstruct_DG(D, k, n, c, p, scheme) for p in np.array_split(pts, len(pts) // 2000 + 1)])


@pytest.mark.parametrize("D,k,n,scheme", CASES)
@pytest.mark.parametrize("count", [4096, 40001])
def test_many_points(sgdg, O, D, k, n, scheme, count):
    rng = np.random.default_rng(D * 100 + k * 10 + n)
    N = sgdg.get_size(D, k, n, scheme)
    c = rng.standard_normal(N)
    pts = np.concatenate([rng.random((count - 400, D)), edge_points(D, n, rng, 300), edge_points(D, n + 3, rng, 100)])
    pts[-1, 0] = 1.0 + 2.0 ** -52  # past the end: zero
    pts[-2, D - 1] = 7.5
    got = sgdg.reconstruct_DG(D, k, n, c, pts, scheme)
    ref = in_parts(sgdg, D, k, n, c, pts, scheme)
    scale = np.max(np.abs(ref))
    assert np.max(np.abs(got - ref)) <= 1e-12 * scale
    few = np.concatenate([pts[:100], pts[-100:]])
    assert np.max(np.abs(np.concatenate([got[:100], got[-100:]]) - O.reconstruct(D, k, n, c, few, scheme))) <= 1e-12 * scale
    assert got[-1] == 0.0 and got[-2] == 0.0


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_coefficients_that_are_not_finite(sgdg, value):
    D, k, n = 2, 3, 6
    rng = np.random.default_rng(0)
    c = rng.standard_normal(sgdg.get_size(D, k, n))
    c[len(c) // 2] = value
    pts = rng.random((20000, D))
    got, ref = sgdg.reconstruct_DG(D, k, n, c, pts), in_parts(sgdg, D, k, n, c, pts, "sparse")
    assert not np.all(np.isfinite(ref))
    assert np.array_equal(got, ref, equal_nan=True)


def test_coordinates_without_a_cell_and_no_room(sgdg):
    D, k, n = 3, 3, 5
    rng = np.random.default_rng(1)
    c = rng.standard_normal(sgdg.get_size(D, k, n))
    pts = rng.random((5000, D))
    ref = sgdg.reconstruct_DG(D, k, n, c, pts)
    for bad in (-1e-300, np.nan):
        p = pts.copy()
        p[4321, 1] = bad
        with pytest.raises(sgdg.SGDGError) as e:
            sgdg.reconstruct_DG(D, k, n, c, p)
        assert e.value.code == 1
    try:  # room for the arguments, not for the pieces: block by block
        sgdg.set_hbm_budget(sgdg.hbm_in_use() + 8 * (c.size + 4 * len(pts)) + 64)
        got = sgdg.reconstruct_DG(D, k, n, c, pts)
    finally:
        sgdg.set_hbm_budget(0)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))

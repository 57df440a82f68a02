"""Values at many points (levels summed along a dimension first) are as near the
exact ones, computed in long double, as those of few points (block by block)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble


def polynomials(k):
    """Legendre polynomials (k, k) and Alpert's wavelets as their left and right halves (2, k, k), orthonormal."""
    p = np.arange(2 * k) % k
    s = np.arange(2 * k) // k
    power = p[:, None] + p[None, :]
    G = np.where(power % 2 == (s[:, None] + s[None, :]) % 2, LD(2) / (1 + power).astype(LD), LD(0))
    unit = np.eye(2 * k, dtype=LD)

    def without(v, others):
        for w in others:
            v = v - (v @ G @ w) * w
        return v
    leg = []
    for j in range(k):
        v = without(unit[j], leg)
        leg.append(v / np.sqrt(v @ G @ v))
    g = [without(unit[k + j], leg) for j in range(k)]
    h = [v.copy() for v in g]
    for i in range(k - 1):
        for j in range(i + 1, k):
            h[j] = h[j] - (h[j] @ G @ unit[k + i]) / (g[i] @ G @ unit[k + i]) * g[i]
    q = [None] * k
    for i in reversed(range(k)):
        v = without(h[i], q[i + 1:])
        q[i] = v / np.sqrt(v @ G @ v)
    q = np.stack(q)
    return np.stack(leg)[:, :k], np.stack([q[:, :k] - q[:, k:], q[:, :k] + q[:, k:]])


def exact(sgdg, D, k, n, c, X):
    leg, wav = polynomials(k)
    tab, cell = {}, {}
    for d in range(D):
        for l in range(n + 1):
            x = X[:, d].astype(LD)
            if l == 0:
                cl, y, poly, scale = np.zeros(len(X), int), 2 * x - 1, [leg, leg], np.sqrt(LD(2))
            else:
                cl = np.floor((1 << (l - 1)) * X[:, d]).astype(int)
                y, poly, scale = (1 << l) * x - (2 * cl + 1), wav, np.sqrt(LD(1 << l))
            v = np.zeros((len(X), k), LD)
            for i in range(k - 1, -1, -1):
                v = v * y[:, None] + np.where((y < 0)[:, None], poly[0][None, :, i], poly[1][None, :, i])
            tab[d, l], cell[d, l] = scale * v, cl
    out, off = np.zeros(len(X), LD), 0
    for t in range((n + 1) ** D):
        L = [t // (n + 1) ** d % (n + 1) for d in range(D)]
        if sum(L) > n:
            continue
        at, stride = np.zeros(len(X), int), 1
        for d in range(D):
            at += cell[d, L[d]] * stride
            stride <<= max(0, L[d] - 1)
        b = c[off:off + stride * k ** D].reshape(stride, -1)[at].astype(LD)
        for d in range(D):
            b = (b.reshape(len(X), -1, k) * tab[d, L[d]][:, None, :]).sum(2)
        out += b[:, 0]
        off += stride * k ** D
    assert off == len(c)
    return out


@pytest.mark.parametrize("D,k,n,points", [(1, 3, 10, 1 << 15), (2, 3, 7, 4096), (3, 3, 6, 4096), (2, 2, 8, 1 << 13)])
def test_many_points_as_near_as_few(sgdg, D, k, n, points):
    # coefficients that decay as those of smooth functions do; 10 % for what the
    # two orders of summation do by chance to a norm over 4096 points and more
    rng = np.random.default_rng(10 * D + k)
    modes = [(tuple(int(v) for v in rng.integers(1, 4, D)), float(rng.uniform(-1, 1)), "sin", 0.3) for _ in range(3)]
    c = sgdg.fourier_coeffs(D, k, n, modes)
    X = rng.random((points, D))
    ref = exact(sgdg, D, k, n, c, X)

    def error(v):
        return float(np.linalg.norm((v - ref).astype(float)))
    few = np.concatenate([sgdg.reconstruct_DG(D, k, n, c, x) for x in np.array_split(X, points // 2048)])
    assert error(few) <= 1e-14 * float(np.linalg.norm(ref.astype(float)))
    assert error(sgdg.reconstruct_DG(D, k, n, c, X)) <= 1.1 * error(few)

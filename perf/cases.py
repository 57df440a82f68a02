"""What this framework is measured on: the work its users have it do.

GalerkinSparseGrids' run time goes into applying the sparse-grid DG derivative
operator, mostly inside fixed-step RK4 time stepping, so that is what most of
the cases do, through the package's public entry points: one operator
application, one solve evolved from host arrays to host arrays (the assembled
FP64 form, which is the default, and the FP32 matrix-free form), batches of
solves that share an operator or have operators of their own, the Vlasov
evolver in both forms, the request server, and the evaluation of a solution at
points.  Sizes are those of the repository's configurations and tests (2D
k=3 n=5; 3D k=3 n=7, alone and 256 at a time; uneven batches of D 2-3, k 2-4,
n 4-7; Vlasov 2x2v k=2 n=8; requests of D 2-4), with smaller ones around them.

Initial data are seeded sums of a few Fourier modes (wave numbers 1..3), what
the repository's workloads start from.  Time steps lie inside RK4's stability
region, so a state can be stepped on for as long as one likes.

exact() states the results in 64 bits with its own construction of the basis,
the 1D operator, the index map and the collocation maps.
"""
import ctypes
import functools
import importlib

import numpy as np
import torch

import __graft_entry__ as entry

DEV = "cuda" if torch.cuda.is_available() else "cpu"


@functools.lru_cache(maxsize=1)
def package():
    return entry.load_package(build=False)


def part(name):
    return importlib.import_module(package().__name__ + "." + name)


# ------------------------------------------------------------------ cases ----
def listed():
    return [
        # one derivative of a small 2D grid: the smallest call, as an energy or a residual makes it
        {"name": "apply_2d", "path": "apply", "D": 2, "k": 3, "n": 5, "which": 1, "method": "plain"},
        # the Laplacian of the 3D wave configuration, once, on vectors the caller keeps on the GPU
        {"name": "apply_laplacian_3d", "path": "apply", "D": 3, "k": 3, "n": 7, "which": 0, "method": "plain"},
        # the small 2D wave evolution, host arrays in and out, the default form: launches and latency
        {"name": "wave_2d", "path": "wave", "D": 2, "k": 3, "n": 5, "nsteps": 200, "nout": 5, "method": "plain"},
        # an advected field in four dimensions, one request served alone by the default form
        {"name": "advect_4d", "path": "advect", "D": 4, "k": 2, "n": 6, "nsteps": 60, "nout": 2, "method": "plain"},
        # an ensemble of 3D waves sharing the assembled operator, FP64 throughout
        {"name": "wave_batch_plain", "path": "plain_batch", "D": 3, "k": 3, "n": 7, "solves": 48, "nsteps": 3},
        # the benchmark's batch: 256 3D waves advanced together, then read back
        {"name": "wave_batch", "path": "batch", "D": 3, "k": 3, "n": 7, "solves": 256, "nsteps": 15},
        # the same batch with its states in pinned host memory before and after every step
        {"name": "wave_batch_host", "path": "batch_host", "D": 3, "k": 3, "n": 7, "solves": 256, "nsteps": 1,
         "chunks": 16},
        # independent advection solves of uneven sizes in the same launches
        {"name": "uneven_batch", "path": "uneven", "solves": 96, "nsteps": 20, "mix": 33},
        # Vlasov transport in 2x2v phase space, the default form
        {"name": "vlasov_2x2v", "path": "vlasov", "D": 2, "k": 2, "n": 8, "nsteps": 8, "method": "plain"},
        # an ensemble of smaller Vlasov problems, matrix-free, in the same launches
        {"name": "vlasov_batch", "path": "vlasov_batch", "D": 2, "k": 2, "n": 6, "solves": 8, "nsteps": 8},
        # a solution sampled at many points (error measures, plots)
        {"name": "evaluate_3d", "path": "evaluate", "D": 3, "k": 3, "n": 7, "points": 1 << 18},
        # a burst of requests through the continuously batching server
        {"name": "serve", "path": "serve", "requests": 8, "mix": 5},
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def _shape(rng, dims, ks, limit, nmin=2, nmax=9):
    """(D, k, n) with at most `limit` coefficients, every refinement that fits equally likely."""
    while True:
        D, k = rng.choice(dims), rng.choice(ks)
        ns = [n for n in range(nmin, nmax + 1) if size(D, k, n) <= limit]
        if ns:
            return D, k, rng.choice(ns)


def draw(rng):
    path = rng.choice(["apply", "wave", "advect", "plain_batch", "batch", "batch_host", "uneven", "vlasov",
                       "vlasov_batch", "evaluate", "serve"])
    method = rng.choice(["plain", "plain", "matfree"])
    if path == "apply":
        D, k, n = _shape(rng, [1, 2, 3, 4], [2, 3, 4], 60000)
        return {"path": path, "D": D, "k": k, "n": n, "which": rng.randint(0, D), "method": method}
    if path == "wave":
        D, k, n = _shape(rng, [1, 2, 3], [2, 3, 4], 46000, nmin=3)
        return {"path": path, "D": D, "k": k, "n": n, "nsteps": _log_int(rng, 20, 200), "nout": rng.randint(2, 5),
                "method": method}
    if path == "advect":
        D, k, n = _shape(rng, [2, 3, 4], [2, 3], 46000, nmin=3)
        return {"path": path, "D": D, "k": k, "n": n, "nsteps": _log_int(rng, 20, 200), "nout": rng.randint(2, 3),
                "method": method}
    if path == "plain_batch":
        D, k, n = _shape(rng, [2, 3], [2, 3, 4], 46000, nmin=4)
        return {"path": path, "D": D, "k": k, "n": n,
                "solves": _log_int(rng, 2, max(2, min(200, 48 * 45792 // size(D, k, n)))), "nsteps": rng.randint(1, 5)}
    if path in ("batch", "batch_host"):
        D, k, n = _shape(rng, [2, 3], [2, 3, 4], 46000, nmin=4)
        case = {"path": path, "D": D, "k": k, "n": n,
                "solves": _log_int(rng, 1, max(1, min(256, 256 * 45792 // size(D, k, n)))),
                "nsteps": _log_int(rng, 2, 15) if path == "batch" else rng.randint(1, 2)}
        if path == "batch_host":
            case["chunks"] = rng.choice([8, 16])
        return case
    if path == "uneven":
        return {"path": path, "solves": _log_int(rng, 4, 96), "nsteps": _log_int(rng, 5, 20),
                "mix": rng.randint(0, 10 ** 6)}
    if path == "vlasov":
        D, k, n = rng.choice([(1, 2, rng.randint(4, 8)), (1, 3, rng.randint(3, 7)), (2, 2, rng.randint(3, 8)),
                              (2, 3, rng.randint(3, 5))])
        return {"path": path, "D": D, "k": k, "n": n, "nsteps": rng.randint(2, 8), "method": method}
    if path == "vlasov_batch":
        D, k, n = rng.choice([(1, 2, rng.randint(4, 8)), (1, 3, rng.randint(3, 7)), (2, 2, rng.randint(3, 6))])
        return {"path": path, "D": D, "k": k, "n": n, "solves": _log_int(rng, 1, 8), "nsteps": rng.randint(2, 8)}
    if path == "evaluate":
        D, k, n = _shape(rng, [1, 2, 3, 4], [2, 3, 4], 46000, nmin=3)
        return {"path": path, "D": D, "k": k, "n": n, "points": _log_int(rng, 100, 1 << 18 if D < 4 else 1 << 16)}
    return {"path": "serve", "requests": rng.randint(2, 8), "mix": rng.randint(0, 10 ** 6)}


# ------------------------------------------------- the grid, in plain numpy ----
@functools.lru_cache(maxsize=256)
def level_tuples(D, n):
    """1-based level tuples with sum <= n + D, dimension 1 fastest."""
    out = []
    for c in range((n + 1) ** D):
        L = [c // (n + 1) ** q % (n + 1) + 1 for q in range(D)]
        if sum(L) <= n + D:
            out.append(tuple(L))
    return out


def cells(L):
    return 1 << max(0, L - 2)


@functools.lru_cache(maxsize=4096)
def size(D, k, n):
    # levels 1 and 2 have one cell, level L has 2^(L-2): counted by the level sum, one dimension at a time
    ways = [1]
    for _ in range(D):
        new = [0] * (n + 1)
        for s, w in enumerate(ways[:n + 1]):
            for l in range(n + 1 - s):
                new[s + l] += w * cells(l + 1)
        ways = new
    return k ** D * sum(ways)


@functools.lru_cache(maxsize=32)
def index_1d(D, k, n):
    """(N, D) 1D index along each dimension and (N, D) 1-based levels of every coefficient: level tuples,
    then cells, then modes, dimension 1 fastest."""
    idx, lev = [], []
    for L in level_tuples(D, n):
        grids = np.meshgrid(*([np.arange(cells(l)) for l in L][::-1] + [np.arange(k)] * D), indexing="ij")
        cell, mode = grids[:D][::-1], grids[D:][::-1]
        i = np.stack([(k * ((cells(l) if l >= 2 else 0) + c) + m).ravel() for l, c, m in zip(L, cell, mode)], 1)
        idx.append(i)
        lev.append(np.tile(np.array(L), (i.shape[0], 1)))
    return np.concatenate(idx), np.concatenate(lev)


def legendre(m):
    return np.polynomial.legendre.leg2poly(np.eye(m + 1)[m]) * np.sqrt((2 * m + 1) / 2.0)


@functools.lru_cache(maxsize=8)
def wavelets(k):
    """Alpert's multiwavelets on [-1, 1]: (2k, k) coefficients of x^i and sgn(x) x^i."""
    e = np.arange(2 * k)
    p, s = e % k, e // k
    odd = (s[:, None] + s[None, :]) % 2
    power = p[:, None] + p[None, :]
    G = np.where(power % 2 == odd, 2.0 / (1 + power), 0.0)  # inner products
    unit = np.eye(2 * k)
    leg = []
    for j in range(k):
        v = unit[j].copy()
        for w in leg:
            v -= (unit[j] @ G @ w) * w
        leg.append(v / np.sqrt(v @ G @ v))
    g = []
    for j in range(k):
        v = unit[k + j].copy()
        for w in leg:
            v -= (unit[k + j] @ G @ w) * w
        g.append(v)
    h = [v.copy() for v in g]
    for i in range(k - 1):
        for j in range(i + 1, k):
            h[j] -= (h[j] @ G @ unit[k + i]) / (g[i] @ G @ unit[k + i]) * g[i]
    q = [None] * k
    for i in reversed(range(k)):
        v = h[i].copy()
        for j in range(i + 1, k):
            v -= (h[i] @ G @ q[j]) * q[j]
        q[i] = v / np.sqrt(v @ G @ v)
    return np.stack(q, 1)


def functions_1d(k, n, x, side):
    """(len(x), k 2^n) values of all 1D basis functions at x, one-sided limits from `side`."""
    x = np.asarray(x, np.float64)
    out = [np.sqrt(2.0) * np.stack([np.polynomial.polynomial.polyval(2 * x - 1, legendre(m)) for m in range(k)], 1)]
    w = wavelets(k)
    for l in range(1, n + 1):
        nc = 1 << (l - 1)
        c = x * nc
        at = np.floor(c) if side > 0 else np.ceil(c) - 1
        at = np.clip(at, 0, nc - 1)
        y = 2.0 * (c - at) - 1.0
        up = (y >= 0) if side > 0 else (y > 0)
        P = y[:, None] ** np.arange(k)[None, :]
        v = np.sqrt(float(1 << l)) * (P @ w[:k] + np.where(up, 1.0, -1.0)[:, None] * (P @ w[k:]))
        block = np.zeros((len(x), nc, k))
        block[np.arange(len(x)), at.astype(int)] = v
        out.append(block.reshape(len(x), nc * k))
    return np.concatenate(out, 1)


@functools.lru_cache(maxsize=32)
def derivative_1d(k, n):
    """The 1D periodic DG derivative with central flux in the hierarchical basis, and its spectral radius."""
    nf = 1 << n
    gx, gw = np.polynomial.legendre.leggauss(k + 1)
    P = [legendre(m) * np.sqrt(2.0) for m in range(k)]  # on [0, 1] of a finest cell
    val = lambda x: np.stack([np.polynomial.polynomial.polyval(2 * x - 1, p) for p in P], 1)  # noqa: E731
    der = lambda x: np.stack([2 * np.polynomial.polynomial.polyval(2 * x - 1, np.polynomial.polynomial.polyder(p))  # noqa: E731
                              if len(p) > 1 else np.zeros_like(x) for p in P], 1)
    t = 0.5 + 0.5 * gx
    here = -(der(t) * (0.5 * gw)[:, None]).T @ val(t)
    a0, a1 = val(np.array([0.0]))[0], val(np.array([1.0]))[0]
    here += 0.5 * np.outer(a1, a1) - 0.5 * np.outer(a0, a0)
    A = np.zeros((nf, k, nf, k))
    for c in range(nf):
        A[c, :, c] += here
        A[c, :, (c + 1) % nf] += 0.5 * np.outer(a1, a0)
        A[c, :, (c - 1) % nf] -= 0.5 * np.outer(a0, a1)
    A = A.reshape(nf * k, nf * k) * nf
    x = ((np.arange(nf)[:, None] + t[None, :]) / nf).ravel()
    F = functions_1d(k, n, x, +1).reshape(nf, k + 1, -1)
    Q = np.einsum("cpj,pm->cmj", F, val(t) * (0.5 * gw)[:, None]).reshape(nf * k, -1) / np.sqrt(float(nf))
    op = Q.T @ (A @ Q)
    op[np.abs(op) < 1e-11 * np.abs(op).max()] = 0.0
    return op, float(np.linalg.norm(op, 2))


@functools.lru_cache(maxsize=32)
def fourier_1d(k, n, a):
    """1D coefficients of exp(2 pi i a x)."""
    gx, gw = np.polynomial.legendre.leggauss(16)
    nf = 2 << n
    x = ((np.arange(nf)[:, None] + 0.5 + 0.5 * gx[None, :]) / nf).ravel()
    w = np.tile(0.5 * gw / nf, nf)
    return functions_1d(k, n, x, +1).T @ (w * np.exp(2j * np.pi * a * x))


def entries(D, k, n):
    """Multiplications one application of all D derivatives needs: the nonzeros of the 1D operator's leading
    blocks, line by line."""
    op, _ = derivative_1d(k, n)
    idx, lev = index_1d(D, k, n)
    lv = np.concatenate([np.full(k * cells(l), l) for l in range(1, n + 2)])
    count = np.stack([(op != 0)[:, lv <= m].sum(1) for m in range(n + 2)], 1)
    lmax = n + D - lev.sum(1)
    return int(sum(count[idx[:, d], lmax + lev[:, d]].sum() for d in range(D)))


def on_lines(D, k, n, d, A):
    """The 1D matrix A along dimension d of the sparse grid (each line its leading block), as a torch CSR matrix."""
    idx, lev = index_1d(D, k, n)
    N = idx.shape[0]
    other = np.zeros(N, np.int64)
    for q in range(D):
        if q != d:
            other = other * (k << n) + idx[:, q]
    order = np.lexsort((idx[:, d], other))
    first = np.empty(N, np.int64)  # where the line of each coefficient starts in that order
    new = np.flatnonzero(np.r_[True, other[order][1:] != other[order][:-1]])
    first[order] = np.repeat(new, np.diff(np.r_[new, N]))
    m = k * (1 << (n + D - lev.sum(1) + lev[:, d] - 1))  # length of the line
    r, c = np.nonzero(A)
    ptr = np.searchsorted(r, np.arange(A.shape[0] + 1))
    i1 = idx[:, d]
    full = ptr[i1 + 1] - ptr[i1]
    rows = np.repeat(np.arange(N), full)
    at = np.arange(full.sum()) - np.repeat(np.cumsum(full) - full, full) + np.repeat(ptr[i1], full)
    keep = c[at] < m[rows]
    rows, at = rows[keep], at[keep]
    cols = order[first[rows] + c[at]]
    crow = np.r_[0, np.cumsum(np.bincount(rows, minlength=N))]
    return torch.sparse_csr_tensor(torch.from_numpy(crow), torch.from_numpy(cols), torch.from_numpy(A[r[at], c[at]]),
                                   size=(N, N), dtype=torch.float64).to(DEV)


@functools.lru_cache(maxsize=8)
def derivatives(D, k, n):
    op, _ = derivative_1d(k, n)
    return [on_lines(D, k, n, d, op) for d in range(D)]


def rk4(f, y, dt, nsteps):
    for _ in range(nsteps):
        k1 = f(y)
        k2 = f(y + 0.5 * dt * k1)
        k3 = f(y + 0.5 * dt * k2)
        y = y + dt / 6.0 * (k1 + 2 * k2 + 2 * k3 + f(y + dt * k3))
    return y


def wave_rhs(D, k, n):
    ops = derivatives(D, k, n)
    N = size(D, k, n)
    return lambda y: torch.cat([y[N:], sum(A @ (A @ y[:N]) for A in ops)])


def advect_rhs(D, k, n, a):
    ops = derivatives(D, k, n)
    return lambda y: -sum(float(v) * (A @ y) for v, A in zip(a, ops))


# ----------------------------------------------------------------- inputs ----
@functools.lru_cache(maxsize=12)
def fields(D, k, n):
    """54 (D = 3: 27 wave vectors, sine and cosine) or fewer Fourier modes as coefficient vectors on the GPU."""
    idx, _ = index_1d(D, k, n)
    rng = np.random.default_rng(77)
    vecs = [np.array([c // 3 ** q % 3 + 1 for q in range(D)]) for c in range(3 ** D)]
    if len(vecs) > 27:
        vecs = [vecs[i] for i in rng.choice(len(vecs), 27, replace=False)]
    at = torch.from_numpy(idx).to(DEV)
    one = [torch.from_numpy(fourier_1d(k, n, a)).to(DEV) for a in (1, 2, 3)]
    out = []
    for v in vecs:
        z = one[v[0] - 1][at[:, 0]]
        for q in range(1, D):
            z = z * one[v[q] - 1][at[:, q]]
        out += [z.real, z.imag]
    return torch.stack(out)


def states(D, k, n, count, rng, nfields=1, modes=6):
    """(count, nfields N) initial states on the GPU, each field a sum of a few seeded modes."""
    F = fields(D, k, n)
    C = np.zeros((count * nfields, F.shape[0]))
    for row in C:
        for j in rng.integers(0, F.shape[0], modes):
            row[j] += rng.uniform(-1, 1)
    return (torch.from_numpy(C).to(DEV) @ F).reshape(count, nfields * F.shape[1])


def wave_dt(D, k, n):
    return 2.0 / (np.sqrt(D) * derivative_1d(k, n)[1])


def advect_dt(k, n, a):
    return 0.5 / (float(np.sum(np.abs(a))) * derivative_1d(k, n)[1])


@functools.lru_cache(maxsize=6)
def operator(D, k, n):
    """The handle a program keeps for its grid."""
    return package().SparseGridOperator(D, k, n)


@functools.lru_cache(maxsize=3)
def vlasov_operator(D, k, n):
    op = package().VlasovOperator(D, k, n)
    op.v_point()  # assembles the operators on the GPU
    return op


def vlasov_inputs(D, k, n, seed):
    F, f0 = part("workloads").vlasov_case(package(), D, k, n, seed=seed)
    dt = 1.0 / (derivative_1d(k, n)[1] * (D + float(np.sum(np.max(np.abs(F), axis=1)))))
    return F, f0, dt


def uneven_specs(case):
    """(D, k, n) of the solves of a mix: a draw of the uneven batch's shapes."""
    rng = np.random.default_rng(case["mix"])
    return [(int(rng.integers(2, 4)), int(rng.integers(2, 5)), int(rng.integers(4, 8))) for _ in range(case["solves"])]


def request_specs(case):
    """(D, k, n, steps) of a burst of requests: the serving stream's shapes, fewer steps."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["requests"]):
        D = int(rng.integers(2, 5))
        out.append((D, int(rng.choice([2, 3])), int(rng.integers(4, 9 if D < 4 else 6)), int(rng.integers(25, 101))))
    return out


def solves_of(specs, rng):
    out = []
    for s in specs:
        a = rng.uniform(-1, 1, s[0])
        out.append((s, a, advect_dt(s[1], s[2], a), states(s[0], s[1], s[2], 1, rng, modes=3)[0].cpu().numpy()))
    return out


def pinned(length):
    return torch.zeros(length, dtype=torch.float64, pin_memory=DEV == "cuda")


def prepare(case, seed):
    sg = package()
    rng = np.random.default_rng(seed)
    path, s = case["path"], {"case": case}
    if path in ("apply", "wave", "advect", "plain_batch", "batch", "batch_host", "evaluate"):
        g = case["D"], case["k"], case["n"]
    if path == "apply":
        s["op"] = operator(*g)
        s["x"] = states(*g, 1, rng)[0]
        s["y"] = torch.zeros_like(s["x"])
    elif path == "wave":
        y0 = states(*g, 1, rng, nfields=2)[0].cpu().numpy()
        s.update(op=operator(*g), f0=y0[:len(y0) // 2], v0=y0[len(y0) // 2:], dt=wave_dt(*g))
    elif path == "advect":
        a = rng.uniform(-1, 1, case["D"])
        s.update(op=operator(*g), f0=states(*g, 1, rng)[0].cpu().numpy(), a=a, dt=advect_dt(g[1], g[2], a))
    elif path == "plain_batch":
        s.update(op=operator(*g), y=states(*g, case["solves"], rng, nfields=2).contiguous(), dt=wave_dt(*g),
                 stream=torch.cuda.Stream())
    elif path in ("batch", "batch_host"):
        y0 = states(*g, case["solves"], rng, nfields=2).cpu()
        b, dt = sg.Batch(), wave_dt(*g)
        for y in y0.numpy():
            b.add("wave", *g, y, dt)
        s.update(batch=b, out=pinned(y0.numel()))
        if path == "batch_host":
            s["in"] = pinned(y0.numel())
            s["in"].copy_(y0.reshape(-1))
        b.step(0)  # the solves move in
    elif path == "uneven":
        s["batch"] = sg.Batch()
        for (D, k, n), a, dt, y in solves_of(uneven_specs(case), rng):
            s["batch"].add("advect", D, k, n, y, dt, a=a)
        s["out"] = pinned(s["batch"].total_size())
        s["batch"].step(0)
    elif path == "vlasov":
        s["op"] = vlasov_operator(case["D"], case["k"], case["n"])
        s["F"], s["f0"], s["dt"] = vlasov_inputs(case["D"], case["k"], case["n"], seed)
    elif path == "vlasov_batch":
        s["batch"] = sg.Batch()
        for j in range(case["solves"]):
            F, f0, dt = vlasov_inputs(case["D"], case["k"], case["n"], 1000 * seed + j)
            s["batch"].add_vlasov(case["D"], case["k"], case["n"], f0, F, dt)
        s["out"] = pinned(s["batch"].total_size())
        s["batch"].step(0)
    elif path == "evaluate":
        s["c"] = states(*g, 1, rng)[0].contiguous()
        s["x"] = torch.from_numpy(rng.random((case["points"], case["D"]))).to(DEV)
        s["v"] = torch.zeros(case["points"], dtype=torch.float64, device=DEV)
    else:
        s["server"] = sg.Server(max_chunk_steps=25)
        s["solves"] = solves_of(request_specs(case), rng)
    return s


# -------------------------------------------------------------------- run ----
def run(s):
    sg = package()
    case = s["case"]
    path = case["path"]
    if path == "apply":
        s["op"].apply_device(s["x"].data_ptr(), s["y"].data_ptr(), which=case["which"], method=case["method"],
                             stream=torch.cuda.current_stream().cuda_stream)
        return s["y"]
    if path == "wave":
        return sg.wave_evolve(case["D"], case["k"], case["n"], s["f0"], s["v0"], 0.0, case["nsteps"] * s["dt"],
                              nsteps=case["nsteps"], nout=case["nout"], method=case["method"], op=s["op"])
    if path == "advect":
        return sg.advect_evolve(case["D"], case["k"], case["n"], s["a"], s["f0"], 0.0, case["nsteps"] * s["dt"],
                                nsteps=case["nsteps"], nout=case["nout"], method=case["method"], op=s["op"])
    if path == "plain_batch":
        s["op"].plain_steps_device(s["y"].data_ptr(), case["solves"], s["dt"], case["nsteps"],
                                   stream=s["stream"].cuda_stream)
        return s["y"]
    if path in ("batch", "uneven", "vlasov_batch"):
        s["batch"].step(case["nsteps"])
        s["batch"].download(s["out"].data_ptr())
        return s["out"]
    if path == "batch_host":
        s["batch"].step_host(s["in"].data_ptr(), s["out"].data_ptr(), case["nsteps"], case["chunks"])
        return s["out"]
    if path == "vlasov":
        return sg.vlasov_evolve(case["D"], case["k"], case["n"], s["F"], s["f0"], 0.0, case["nsteps"] * s["dt"],
                                nsteps=case["nsteps"], op=s["op"], method=case["method"])
    if path == "evaluate":
        sg.check(sg.lib().sgdg_evaluate_device(case["D"], case["k"], case["n"], 0, ctypes.c_void_p(s["c"].data_ptr()),
                                               case["points"], ctypes.c_void_p(s["x"].data_ptr()),
                                               ctypes.c_void_p(s["v"].data_ptr()),
                                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return s["v"]
    srv = s["server"]
    ids = [srv.submit("advect", q[0], q[1], q[2], y, dt, q[3], a=a) for q, a, dt, y in s["solves"]]
    while any(srv.status(i)[0] in (srv.QUEUED, srv.RUNNING) for i in ids):
        srv.tick()
    return [srv.result(i, v[3].size) for i, v in zip(ids, s["solves"])]


# ------------------------------------------------------------------- work ----
def work(case):
    """Bytes: a step reads the stage inputs and the FP64 state and accumulator and writes them once per stage,
    32 bytes per coefficient and stage, beside what goes in and comes out; one application reads and writes a
    vector.  The operator is a 1D table.  Operations: a multiplication and an addition per nonzero of the 1D
    operator along every line (the Laplacian applies each derivative twice)."""
    path = case["path"]
    if path == "apply":
        D, k, n = case["D"], case["k"], case["n"]
        e = entries(D, k, n) * (2 if case["which"] == 0 else 1 / D)
        return {"bytes": 16 * size(D, k, n), "flops": 2 * e}
    if path in ("wave", "plain_batch", "batch", "batch_host"):
        D, k, n, c = case["D"], case["k"], case["n"], case.get("solves", 1)
        N = 2 * size(D, k, n)
        moved = {"wave": 8 * N * (1 + case.get("nout", 0)), "plain_batch": 0, "batch": 8 * N, "batch_host": 16 * N}[path]
        return {"bytes": c * (128 * N * case["nsteps"] + moved),
                "flops": c * 4 * case["nsteps"] * (4 * entries(D, k, n) + 7 * N)}
    if path == "advect":
        D, k, n = case["D"], case["k"], case["n"]
        N = size(D, k, n)
        return {"bytes": 128 * N * case["nsteps"] + 8 * N * (1 + case["nout"]),
                "flops": 4 * case["nsteps"] * (2 * entries(D, k, n) + 7 * N)}
    if path in ("uneven", "serve"):
        specs = [q + (case["nsteps"],) for q in uneven_specs(case)] if path == "uneven" else request_specs(case)
        return {"bytes": sum(size(*q[:3]) * (128 * q[3] + 16) for q in specs),
                "flops": sum(4 * q[3] * (2 * entries(*q[:3]) + 7 * size(*q[:3])) for q in specs)}
    if path in ("vlasov", "vlasov_batch"):
        P, k, n, c = 2 * case["D"], case["k"], case["n"], case.get("solves", 1)
        N = size(P, k, n)
        # per stage the P derivatives, both maps of each and both maps back, a triangular 1D map
        # (a block a level) along every dimension each
        maps = 2 * P * (P + 1) * N * k * (n + 2) / 2
        return {"bytes": c * case["nsteps"] * 4 * N * (32 + 8 * P), "flops": c * case["nsteps"] * 8 * (entries(P, k, n) + maps)}
    D, k, n, pts = case["D"], case["k"], case["n"], case["points"]
    return {"bytes": 8 * (size(D, k, n) + pts * (D + 1)), "flops": 2.0 * pts * len(level_tuples(D, n)) * k ** D}


# ------------------------------------------------------------------ exact ----
@functools.lru_cache(maxsize=4)
def collocation(k, n):
    """(U, L): the values of the 1D basis functions at the collocation points are L U, L unit lower and U upper
    triangular in the levels."""
    from_right, from_left = [], []
    for l in range(n + 1):
        nc = 1 << max(0, l - 1)
        for c in range(nc):
            for t in range(k - 1):
                node = t / (k - 1) if l == 0 else (2 * t + 1) / (2 * (k - 1))
                from_right.append((len(from_right) + len(from_left), (c + node) / nc))
            from_left.append((len(from_right) + len(from_left), 1.0 if l == 0 else (c + 0.5) / nc))
    V = np.zeros((k << n, k << n))
    for pts, side in ((from_right, +1), (from_left, -1)):
        V[[i for i, _ in pts]] = functions_1d(k, n, np.array([x for _, x in pts]), side)
    coords = np.zeros(k << n)
    for i, x in from_right + from_left:
        coords[i] = x
    U, low = V.copy(), np.eye(k << n)
    at = 0
    for l in range(n):
        to = at + k * (1 << max(0, l - 1))
        f = np.linalg.solve(U[at:to, at:to].T, U[to:, at:to].T).T
        f[np.abs(f) < 1e-13] = 0.0
        low[to:, at:to] = f
        U[to:] -= f @ U[at:to]
        U[to:, at:to] = 0.0
        at = to
    U[np.abs(U) < 1e-12] = 0.0
    return U, low, coords


def vlasov_exact(D, k, n, F, f0, dt, nsteps):
    P = 2 * D
    U, low, coords = collocation(k, n)
    clean = lambda A: np.where(np.abs(A) < 1e-13, 0.0, A)  # noqa: E731
    maps = [[on_lines(P, k, n, d, A) for d in range(P)]
            for A in (U, low, clean(np.linalg.inv(low)), clean(np.linalg.inv(U)))]
    ops = derivatives(P, k, n)
    idx, _ = index_1d(P, k, n)
    v = torch.from_numpy(2 * coords[idx[:, D:]] - 1).to(DEV)
    F = torch.from_numpy(F).to(DEV)

    def through(x, *which):
        for w in which:
            for A in maps[w]:
                x = A @ x
        return x

    def rhs(f):
        p = torch.stack([A @ f for A in ops], 1)
        p = through(p, 0, 1)
        return through(-(v * p[:, :D]).sum(1) + (F.T * p[:, D:]).sum(1), 2, 3)
    return rk4(rhs, torch.from_numpy(f0).to(DEV), dt, nsteps).cpu().numpy()


def evaluate_exact(D, k, n, c, x):
    tables, at, off = [], [], 0
    w = torch.from_numpy(wavelets(k)).to(DEV)
    for d in range(D):
        vs, cs = [], []
        for l in range(n + 1):
            if l == 0:
                vs.append(np.sqrt(2.0) * torch.stack([sum(float(a) * (2 * x[:, d] - 1) ** i for i, a in enumerate(legendre(m)))
                                                      for m in range(k)], 1))
                cs.append(torch.zeros(x.shape[0], dtype=torch.int64, device=x.device))
                continue
            nc = 1 << (l - 1)
            cell = torch.clamp(torch.floor(nc * x[:, d]), max=nc - 1)
            y = 2.0 * (nc * x[:, d] - cell) - 1.0
            Y = torch.stack([y ** i for i in range(k)], 1)
            vs.append(np.sqrt(float(1 << l)) * (Y @ w[:k] + torch.where(y >= 0, 1.0, -1.0).double()[:, None] * (Y @ w[k:])))
            cs.append(cell.long())
        tables.append(vs)
        at.append(cs)
    out = torch.zeros(x.shape[0], dtype=torch.float64, device=x.device)
    for L in level_tuples(D, n):
        cl, stride = torch.zeros(x.shape[0], dtype=torch.int64, device=x.device), 1
        for d in range(D):
            cl = cl + at[d][L[d] - 1] * stride
            stride *= cells(L[d])
        t = c[off:off + stride * k ** D].reshape(stride, -1)[cl]
        for d in range(D):  # the fastest mode is the first dimension's
            t = (t.reshape(x.shape[0], -1, k) * tables[d][L[d] - 1][:, None, :]).sum(2)
        out += t[:, 0]
        off += stride * k ** D
    return out


def exact(case, seed):
    rng = np.random.default_rng(seed)
    path = case["path"]
    if path in ("apply", "wave", "advect", "plain_batch", "batch", "batch_host", "evaluate"):
        g = case["D"], case["k"], case["n"]
    if path == "apply":
        x = states(*g, 1, rng)[0]
        ops = derivatives(*g)
        return sum(A @ (A @ x) for A in ops) if case["which"] == 0 else ops[case["which"] - 1] @ x
    if path in ("wave", "advect"):
        if path == "wave":
            y, dt = states(*g, 1, rng, nfields=2)[0], wave_dt(*g)
            f = wave_rhs(*g)
        else:
            a = rng.uniform(-1, 1, case["D"])
            y, dt, f = states(*g, 1, rng)[0], advect_dt(g[1], g[2], a), advect_rhs(*g, a)
        out, done, ns, nout = [], 0, case["nsteps"], case["nout"]
        at = [ns * i // (nout - 1) for i in range(nout)]
        for i in at:
            y = rk4(f, y, dt, i - done)
            done = i
            out.append(y.cpu().numpy())
        return np.array([ns * dt * i / ns for i in at]), out
    if path in ("plain_batch", "batch", "batch_host"):
        y = states(*g, case["solves"], rng, nfields=2)
        y = rk4(wave_rhs(*g), y.T.contiguous(), wave_dt(*g), case["nsteps"]).T.contiguous()
        return y if path == "plain_batch" else y.reshape(-1).cpu()
    if path in ("uneven", "serve"):
        specs = uneven_specs(case) if path == "uneven" else request_specs(case)
        out = [rk4(advect_rhs(*q[:3], a), torch.from_numpy(y).to(DEV), dt, case["nsteps"] if path == "uneven" else q[3]).cpu()
               for q, a, dt, y in solves_of(specs, rng)]
        return torch.cat(out) if path == "uneven" else [y.numpy() for y in out]
    if path == "vlasov":
        F, f0, dt = vlasov_inputs(case["D"], case["k"], case["n"], seed)
        return (np.array([0.0, case["nsteps"] * dt]),
                [f0, vlasov_exact(case["D"], case["k"], case["n"], F, f0, dt, case["nsteps"])])
    if path == "vlasov_batch":
        return torch.cat([torch.from_numpy(vlasov_exact(case["D"], case["k"], case["n"], *vlasov_inputs(
            case["D"], case["k"], case["n"], 1000 * seed + j), case["nsteps"])) for j in range(case["solves"])])
    c = states(*g, 1, rng)[0]
    x = torch.from_numpy(rng.random((case["points"], case["D"]))).to(DEV)
    return evaluate_exact(*g, c, x)

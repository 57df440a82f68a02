"""A re-plan after a change of stream, or after replays of a captured step on
another stream, with that work still in flight: it ends before its memory is
moved and reused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D, k, n, dt = 3, 3, 6, 1e-4


def solves(sgdg, count, seed=0):
    N = 2 * sgdg.get_size(D, k, n)
    return np.random.default_rng(seed).standard_normal((count, N))


def alone(sgdg, y0, steps):
    b = sgdg.Batch()
    i = b.add("wave", D, k, n, y0, dt)
    b.step(steps)
    out = b.state(i)
    b.close()
    return out


@pytest.mark.parametrize("others", [False, True])
def test_join_on_another_stream(sgdg, others):
    import torch
    y = solves(sgdg, 9)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    b = sgdg.Batch()
    b.set_stream(s1.cuda_stream)
    ids = [b.add("wave", D, k, n, v, dt) for v in y[:8]]
    b.step(200)  # tens of milliseconds
    ids.append(b.add("wave", D, k, n, y[8], dt))
    if others:  # a class of its own, whose arena is a new one
        b.add("advect", 2, 2, 5, solves(sgdg, 1)[0][:sgdg.get_size(2, 2, 5)], dt, a=[0.5, 0.25])
    b.set_stream(s2.cuda_stream)
    b.step(3)
    got = [b.state(i) for i in ids]
    b.close()
    for i, v in enumerate(y):
        assert np.array_equal(got[i], alone(sgdg, v, 203 if i < 8 else 3)), i


def test_join_after_replays_elsewhere(sgdg):
    import torch
    y = solves(sgdg, 5, 1)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    b = sgdg.Batch()
    b.set_stream(s1.cuda_stream)
    ids = [b.add("wave", D, k, n, v, dt) for v in y[:4]]
    b.step(1)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s1):
        b.step(2)
    with torch.cuda.stream(s2):
        for _ in range(50):
            graph.replay()
    ids.append(b.add("wave", D, k, n, y[4], dt))
    b.step(2)
    got = [b.state(i) for i in ids]
    b.close()
    for i, v in enumerate(y):
        assert np.array_equal(got[i], alone(sgdg, v, 103 if i < 4 else 2)), i

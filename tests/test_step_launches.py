"""Steps launched one after another: every launch leaves the work list's counters
clear for the next, however the steps are split over calls and streams."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,D,k,n,solves", [("wave", 2, 3, 5, 1), ("advect", 3, 2, 6, 40), ("wave", 3, 3, 5, 9)])
def test_steps_split_over_calls_and_streams(sgdg, kind, D, k, n, solves):
    import torch
    rng = np.random.default_rng(solves)
    N = sgdg.get_size(D, k, n) * (2 if kind == "wave" else 1)
    y0, a = rng.standard_normal((solves, N)), rng.uniform(-1, 1, D)

    def run(splits, streams=()):
        b = sgdg.Batch()
        ids = [b.add(kind, D, k, n, y, 1e-4, a=a) for y in y0]
        for i, s in enumerate(splits):
            if streams:
                torch.cuda.synchronize()  # the engine's work moves to another stream
                b.set_stream(streams[i % len(streams)])
            b.step(s)
        out = np.stack([b.state(i) for i in ids])
        b.close()
        return out
    ref = run([1] * 12)
    assert np.array_equal(run([12]), ref)
    assert np.array_equal(run([5, 0, 1, 6]), ref)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    assert np.array_equal(run([3, 4, 5], [s1.cuda_stream, s2.cuda_stream]), ref)
    b = sgdg.Batch()  # from host states, in chunks, two steps a call
    for y in y0:
        b.add(kind, D, k, n, np.zeros(N), 1e-4, a=a)
    h = y0.reshape(-1).copy()
    for _ in range(6):
        b.step_host(h, nsteps=2, chunks=3)
    assert np.array_equal(h.reshape(solves, N), ref)
    b.close()

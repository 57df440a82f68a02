"""Device blocks kept between calls: they count against the HBM budget, are
given back, and several threads with handles of their own share them."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_kept_blocks_are_bounded_and_given_back(sgdg):
    import torch
    torch.zeros(1, device="cuda")
    op = sgdg.SparseGridOperator(3, 3, 6)
    y = torch.zeros(192 * 2 * op.N, dtype=torch.float64, device="cuda")
    op.plain_steps_device(y.data_ptr(), 1, 1e-3, 1)  # the operator
    before = free_bytes()
    in_use = sgdg.hbm_in_use()
    for solves in (192, 150, 192, 96, 130):  # four blocks of up to 57 MB a call
        op.plain_steps_device(y.data_ptr(), solves, 1e-3, 1)
    assert sgdg.hbm_in_use() == in_use  # what is kept is not in use
    held = before - free_bytes()
    assert 0 < held <= (1 << 30) + (8 << 20)
    try:  # a budget without room for it
        sgdg.set_hbm_budget(in_use + 4096)
        assert before - free_bytes() <= 8 << 20
        with pytest.raises(sgdg.SGDGError) as e:
            op.plain_steps_device(y.data_ptr(), 192, 1e-3, 1)
        assert e.value.code == 2
        sgdg.set_hbm_budget(in_use + 5 * 8 * 192 * 2 * op.N)
        op.plain_steps_device(y.data_ptr(), 192, 1e-3, 1)
        op.plain_steps_device(y.data_ptr(), 96, 1e-3, 1)  # other sizes within the budget
        assert before - free_bytes() <= 5 * 8 * 192 * 2 * op.N + (8 << 20)
    finally:
        sgdg.set_hbm_budget(0)
    op.close()


def test_threads_with_handles_of_their_own(sgdg):
    D, k, n, dt, steps = 2, 3, 5, 1e-3, 24
    rng = np.random.default_rng(0)
    N = sgdg.get_size(D, k, n)
    y0 = rng.standard_normal((4, 2 * N))

    def evolve(y, method):
        _, st = sgdg.wave_evolve(D, k, n, y[:N], y[N:], 0.0, steps * dt, nsteps=steps, method=method)
        return st[-1]
    methods = ["plain", "matfree", "plain", "matfree"]
    ref = [evolve(y, m) for y, m in zip(y0, methods)]
    bad = []

    def work(i):
        try:
            for _ in range(20):
                if not np.array_equal(evolve(y0[i], methods[i]), ref[i]):
                    bad.append(i)
        except Exception as e:  # reported by the main thread
            bad.append(e)
    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad

"""Solves that share an operator and a call: one that is not finite is repeated
with the whole operator, and the others' results stay what they are without it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,k,n", [(2, 3, 4), (1, 2, 3)])
@pytest.mark.parametrize("solves,bad", [(1, [0]), (2, [1]), (9, [0]), (9, [3, 4]), (9, [2, 8]), (5, [0, 1, 2, 3, 4])])
@pytest.mark.parametrize("steps", [2, 257])
def test_a_solve_does_not_depend_on_its_neighbours(sgdg, D, k, n, solves, bad, steps):
    import torch
    op = sgdg.SparseGridOperator(D, k, n)
    y = np.random.default_rng(solves).standard_normal((solves, 2 * op.N))

    def step(z):
        dev = torch.tensor(z, device="cuda")
        op.plain_steps_device(dev.data_ptr(), len(z), 1e-5, steps)
        return dev.cpu().numpy()
    fine = step(y)
    for j, i in enumerate(bad):
        y[i, j] = (np.nan, np.inf)[j % 2]
    got = step(y)
    for i in range(solves):
        if i in bad:
            assert not np.all(np.isfinite(got[i]))
            assert np.array_equal(got[i], step(y[i:i + 1])[0], equal_nan=True), i
        else:
            assert np.array_equal(got[i], fine[i]), i
    op.close()


def test_no_room_beside_the_states_of_the_start(sgdg):
    # the repetition fits without them only: all solves with the whole operator
    import torch
    op = sgdg.SparseGridOperator(2, 3, 5)
    y = np.random.default_rng(0).standard_normal((64, 2 * op.N))
    one = torch.tensor(y, device="cuda")
    op.plain_steps_device(one.data_ptr(), 64, 1e-5, 2)
    y[:, 3] = np.nan
    y[5, 3] = 0.25
    two = torch.tensor(y, device="cuda")
    op.device_csr(-1)
    block = 8 * y.size
    ran = []
    try:
        for extra in range(2 * block, 6 * block, block // 2):
            sgdg.set_hbm_budget(sgdg.hbm_in_use() + extra + 1024)
            three = two.clone()
            try:
                op.plain_steps_device(three.data_ptr(), 64, 1e-5, 2)
            except sgdg.SGDGError as e:
                assert e.code == 2 and extra < 3 * block
                assert torch.equal(three.nan_to_num(7.0), two.nan_to_num(7.0))
                continue
            ran.append(extra)
            bad = ~torch.isfinite(three).all(dim=1)
            assert bad.sum() == 63 and not bool(bad[5])
    finally:
        sgdg.set_hbm_budget(0)
    assert len(ran) >= 4
    op.close()

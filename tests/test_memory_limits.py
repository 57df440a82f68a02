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

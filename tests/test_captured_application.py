"""Applications captured in a graph: a replay's result does not depend on what an
earlier replay met, and what the graph uses stays there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def setup(sgdg):
    import torch
    op = sgdg.SparseGridOperator(4, 2, 6)  # large enough for the pruned operator
    x = torch.tensor(np.random.default_rng(0).standard_normal(op.N), device="cuda")
    y = torch.zeros_like(x)
    op.apply_device(x.data_ptr(), y.data_ptr(), which=0)
    torch.cuda.synchronize()
    return torch, op, x, y


def test_replays_on_either_side_of_a_nan(sgdg):
    torch, op, x, y = setup(sgdg)
    called = y.clone()
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        op.apply_device(x.data_ptr(), y.data_ptr(), which=0, stream=s.cuda_stream)
    keep = float(x[5])
    for value in (keep, np.nan, keep, np.inf, keep):
        x[5] = value
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        if value == keep:
            assert torch.equal(y, called)
        else:
            assert not bool(torch.isfinite(y).all())
    op.close()


def test_more_captured_calls_than_words(sgdg):
    torch, op, x, y = setup(sgdg)
    called = y.clone()
    out = torch.zeros(4, op.N, dtype=torch.float64, device="cuda")
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        for i in range(1030):
            op.apply_device(x.data_ptr(), out[i % 4].data_ptr(), which=0, stream=s.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    for i in range(4):  # the last ones with the whole operator
        assert float((out[i] - called).norm()) <= 1e-10 * float(called.norm())
    op.close()


def test_the_operator_stays_for_the_graph(sgdg):
    torch, op, x, y = setup(sgdg)
    called = y.clone()
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        op.apply_device(x.data_ptr(), y.data_ptr(), which=0, stream=s.cuda_stream)
    try:
        sgdg.set_hbm_budget(sgdg.hbm_in_use() + 64)  # every kept operator is asked back
        with pytest.raises(sgdg.SGDGError):
            op.apply(x.cpu().numpy(), 0)
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, called)
        # with a budget a call is captured with the whole operator
        other = torch.cuda.CUDAGraph()
        with torch.cuda.graph(other, stream=s):
            op.apply_device(x.data_ptr(), y.data_ptr(), which=0, stream=s.cuda_stream)
        other.replay()
        torch.cuda.synchronize()
        assert float((y - called).norm()) <= 1e-10 * float(called.norm())
    finally:
        sgdg.set_hbm_budget(0)
    op.close()

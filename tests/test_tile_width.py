"""Widths of the matrix-free tiles without a tuned shape: no wider than their
columns, narrower where a step holds few items per phase, and the same results
at every width."""
import numpy as np
import pytest

from test_worklist import ADVECT, VLASOV, WAVE, check_coverage, check_rk_once, check_schedule, check_stages, dryrun

# alone (narrowest), a few (in between or either end), enough to fill the GPU
BATCHES = [[(WAVE, 3, 3, 5, 0, 1, 0, 0)], [(WAVE, 2, 3, 5, 0, 1, 0, 0)], [(WAVE, 3, 4, 4, 0, 6, 0, 0)],
           [(ADVECT, 3, 2, 5, 0, 90, 0, 0), (ADVECT, 2, 5, 3, 0, 3, 0, 0)], [(VLASOV, 2, 3, 4, 0, 2, 0, 0)],
           [(ADVECT, 2, 1, 4, 1, 2, 0, 0)], [(WAVE, 3, 3, 5, 0, 64, 0, 0)]]


@pytest.mark.parametrize("batch", range(len(BATCHES)))
def test_widths_of_untuned_tiles(sgdg, batch):
    sgdg.clear_tile_shapes()
    it, spec, cls, boff, nctr = dryrun(sgdg, BATCHES[batch])
    check_schedule(it, nctr)
    check_coverage(it, spec, cls, boff)
    check_stages(it)
    check_rk_once(it, spec, cls, boff)
    k = np.array([spec[c][2] for c in it["cls"]])
    cpt = np.where(k <= 3, 4, 2)
    assert np.all(it["W"] >= cpt) and np.all(it["W"] & (it["W"] - 1) == 0)
    assert np.all(it["Wv"] <= it["W"])
    assert np.all((it["W"] == cpt) | (it["W"] // 2 < it["Wv"]))  # no wider than its columns


@pytest.mark.parametrize("big,small", [(40, 60), (64, 1), (3, 90)])
def test_list_order_of_uneven_groups(sgdg, big, small):
    # groups of very different lengths, in list order (the first two) and in
    # wavefronts: either way a schedule whose waits point backwards and whose
    # phases cover every element once
    sgdg.clear_tile_shapes()
    batch = [(ADVECT, 3, 4, 5, 0, big, 0, 0), (ADVECT, 2, 3, 4, 0, small, 0, 0), (WAVE, 2, 2, 5, 0, small, 0, 0),
             (ADVECT, 1, 3, 6, 0, 2, 0, 0)]
    it, spec, cls, boff, nctr = dryrun(sgdg, batch)
    check_schedule(it, nctr)
    check_coverage(it, spec, cls, boff)
    check_stages(it)
    check_rk_once(it, spec, cls, boff)


def test_width_follows_the_items_per_phase(sgdg):
    sgdg.clear_tile_shapes()
    widest = []
    for solves in (1, 16, 64):
        it, *_ = dryrun(sgdg, [(WAVE, 3, 3, 7, 0, solves, 0, 0)])
        widest.append(int(it["W"][it["lmax"] == 8].max()))
    # lines of 128 row blocks: 2^w times 8 columns, w = -2, -1, 0, at least 4
    assert widest == [4, 4, 8]
    it, *_ = dryrun(sgdg, [(WAVE, 3, 3, 7, 0, 1, 0, 0)])
    assert int(it["W"][it["lmax"] == 4].max()) == 32  # 8 row blocks: 128 columns at w = 0
    try:  # a tuned shape is used as it is
        sgdg.set_tile_shape(3, 3, 0, 4)
        it, *_ = dryrun(sgdg, [(WAVE, 3, 3, 7, 0, 1, 0, 0)])
        assert int(it["W"][it["lmax"] == 4].max()) == 128
    finally:
        sgdg.clear_tile_shapes()


@pytest.mark.gpu
def test_results_do_not_depend_on_the_width(sgdg):
    rng = np.random.default_rng(0)
    specs = [("wave", 3, 3, 5), ("advect", 2, 4, 5), ("advect", 3, 2, 4), ("wave", 2, 5, 4)]
    y0 = [rng.standard_normal(sgdg.get_size(D, k, n) * (2 if kind == "wave" else 1)) for kind, D, k, n in specs]
    a = rng.uniform(-1, 1, 3)

    def run():
        b = sgdg.Batch()
        ids = [b.add(kind, D, k, n, y, 1e-4, a=a[:D] if kind == "advect" else None)
               for (kind, D, k, n), y in zip(specs, y0)]
        b.step(7)
        out = [b.state(i) for i in ids]
        b.close()
        return out
    try:
        sgdg.clear_tile_shapes()
        ref = run()
        for wlog in (-2, -1, 0, 2):
            for _, D, k, _ in specs:
                sgdg.set_tile_shape(D, k, wlog, 4)
            for got, want in zip(run(), ref):
                assert np.array_equal(got, want), wlog
    finally:
        sgdg.clear_tile_shapes()

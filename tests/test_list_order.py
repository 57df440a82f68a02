"""The work list in list order: the order that a scan of every group for every
item gives, at a cost per item that does not grow with the groups."""
import ctypes
import heapq
import time

import numpy as np
import pytest

from test_worklist import ADVECT, WAVE, dryrun

CTAS = 456


def scan_order(it, spec):
    """Per item of the list the group that a free CTA takes: most work ahead
    among those that need not wait, else the shortest wait.  One group per class."""
    groups = []
    for c in range(len(spec)):
        idx = np.nonzero(it["cls"] == c)[0]
        kind, _, k = (int(v) for v in spec[c][:3])
        e = it["W"][idx].astype(float) * k * 2.0 ** (it["lmax"][idx] - 1)
        rk = np.where(it["flags"][idx] & 4, 4.0, 0.0)
        cost = 8000.0 + e * (4.0 + 0.7 * k * (2 if kind == WAVE else 1) + rk)
        cuts = np.nonzero(np.diff(it["done_ctr"][idx]))[0] + 1
        phases = np.split(cost, cuts)
        ahead = [0.0]
        for p in reversed(phases):
            ahead.append(ahead[-1] + max(p.max(), p.sum() / CTAS))
        groups.append({"p": phases, "ahead": ahead[::-1], "ph": 0, "i": 0, "ready": 0.0, "done": 0.0})
    ctas = [0.0] * CTAS
    order = []
    for _ in range(len(it["cls"])):
        t = heapq.heappop(ctas)
        best = None
        for g, s in enumerate(groups):
            while s["ph"] < len(s["p"]) and s["i"] == len(s["p"][s["ph"]]):
                s["ready"] = max(s["ready"], s["done"])
                s["ph"] += 1
                s["i"] = 0
            if s["ph"] == len(s["p"]):
                continue
            key = (max(0.0, s["ready"] - (t + 0.65 * s["p"][s["ph"]][s["i"]])), -s["ahead"][s["ph"]])
            if best is None or key < best[0]:
                best = (key, g)
        s = groups[best[1]]
        c = s["p"][s["ph"]][s["i"]]
        s["i"] += 1
        end = max(t + 0.65 * c, s["ready"]) + 0.35 * c
        s["done"] = max(s["done"], end)
        heapq.heappush(ctas, end)
        order.append(best[1])
    return order


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_list_order_is_the_scans(sgdg, seed):
    sgdg.clear_tile_shapes()
    rng = np.random.default_rng(seed)
    batch = [(int(rng.choice([ADVECT, WAVE])), int(rng.integers(2, 4)), int(rng.integers(2, 5)),
              int(rng.integers(4, 7)), 0, 1, 0, 0) for _ in range(24)]
    it, spec, *_ = dryrun(sgdg, batch)
    got = it["cls"].tolist()
    assert got != sorted(got) and len(got) > 300 * 12  # in list order
    assert got == scan_order(it, spec)


def test_cost_per_item_does_not_grow_with_the_groups(sgdg):
    # ten times the groups and the items: a scan of the groups for every item
    # takes eleven times as long for each; room for the heaps' depth and a busy machine
    sgdg.clear_tile_shapes()
    L = sgdg.lib()

    def per_item(groups):
        spec = np.array([(ADVECT, 2, 2, 6, 0, 1, 0, -1)] * groups, dtype=np.int32)
        ni, nb, nc = ctypes.c_int64(), ctypes.c_int64(), ctypes.c_int()
        best = np.inf
        for _ in range(9):
            t = time.perf_counter()
            assert L.sgdg_worklist_dryrun(groups, spec.ctypes.data, 0, 0, 1, None, 0, ctypes.byref(ni),
                                          ctypes.byref(nc), None, None, 0, ctypes.byref(nb)) == 0
            best = min(best, time.perf_counter() - t)
        return best / ni.value
    assert per_item(200) <= 4 * per_item(20)

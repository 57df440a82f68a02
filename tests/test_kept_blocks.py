"""Device blocks kept between calls go with the last handle, also when the tables
of a point evaluation stay for the process."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import numpy as np, torch
import __graft_entry__ as g
sg = g.load_package(build=True)
torch.zeros(1, device="cuda")

def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]
rng = np.random.default_rng(0)
op = sg.SparseGridOperator(3, 3, 6)
assert np.isfinite(sg.reconstruct_DG(3, 3, 4, rng.standard_normal(sg.get_size(3, 3, 4)), [0.25, 0.5, 0.75]))
b = sg.Batch()  # kernels of both forms are loaded before the first measurement
i = b.add("wave", 3, 3, 4, rng.standard_normal(2 * sg.get_size(3, 3, 4)), 1e-4)
b.step(1)
b.state(i)
b.close()
y = torch.zeros(192 * 2 * op.N, dtype=torch.float64, device="cuda")
op.plain_steps_device(y.data_ptr(), 1, 1e-4, 1)
op.close()
before = free()
for close in (True, False):
    op = sg.SparseGridOperator(3, 3, 6)
    op.plain_steps_device(y.data_ptr(), 192, 1e-4, 1)  # four blocks of 57 MB
    assert before - free() > 200 << 20
    if close:
        op.close()
    else:
        sg.set_hbm_budget(0)
    left = before - free()
    assert left < (8 << 20) + (0 if close else 32 << 20), left  # (the operator's own)
"""


def test_blocks_go_with_the_last_handle():
    r = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr

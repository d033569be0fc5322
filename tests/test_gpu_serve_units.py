"""Units of the request server that the split contractions do not take: they run
in FP64, and reserve what that uses."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
import so3_b200 as so3
from so3_b200 import serve
from tests.conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["inverse", "forward"])
def test_small_units_reserve_no_split_scratch(kind):
    n, batch = 32, 4
    p = so3.SO3Parameters(L=128, N=16)
    size = {"inverse": (so3.flmn_size(p), so3.f_size(p)), "forward": (so3.f_size(p), so3.flmn_size(p))}[kind]
    x = torch.randn(2 * size[0], dtype=torch.float64, device="cuda").view(-1, 2)
    x = torch.view_as_complex(x)
    outs = [torch.empty(size[1], dtype=torch.complex128, device="cuda") for _ in range(n)]
    torch.cuda.synchronize()
    with serve.Server(0, memory_budget=8 << 30, max_inflight=1, max_batch=batch, max_L=128) as sv:
        ids = [sv.submit(kind, p, x, o, "mixed") for o in outs]
        res = [sv.wait(i) for i in ids]
        peak = sv.stats()["peak_bytes"]
    torch.cuda.synchronize()
    assert all(r.status == 0 for r in res) and max(r.batch for r in res) == batch
    assert all(torch.equal(torch.view_as_real(o), torch.view_as_real(outs[0])) for o in outs)
    scratch = so3.api.workspace_size(p)  # 33 MB; the split operand of a tile would be 235 MB
    assert peak < batch * (scratch + 16 * (size[0] + size[1])) + (64 << 20)


CODE = """
import torch
import so3_b200 as so3
from so3_b200 import serve
ctx = so3.Context(0)
p = so3.SO3Parameters(L=300, N=2)  # Delta to l = 511: what the table of L = 512, N = 64 is built from
ctx.inverse(torch.zeros(so3.flmn_size(p), dtype=torch.complex128, device="cuda"), p)
torch.cuda.synchronize()
trace = serve.make_trace(40, rate=1e5, seed=21, L_range=(24, 40), N_max=6, p_inverse=1.0, precision="mixed")
with serve.Server(0, memory_budget=8 << 30, max_inflight=2, max_batch=16, max_L=64) as sv:
    res, _, _ = serve.replay(sv, trace)
    assert sv.stats()["peak_bytes"] <= 8 << 30
assert max(r.batch for r in res) >= 8
assert all(r.status == 0 for r in res), [r.status for r in res]
"""


def test_a_split_unit_builds_no_table_beyond_the_budget():
    """The 24 GB digit table does not fit an 8 GB budget: built all the same, it
    would leave every later request without room."""
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, env=dict(os.environ, PYTHONPATH=ROOT),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]

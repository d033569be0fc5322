"""The first transform of a length in a process, on a stream that does not wait
for the legacy one, while large copies keep the copy engines busy: its tables
must be complete before a kernel reads them (the lengths of
test_gpu_table_upload.py, which other tests of one process may have built)."""
import os
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import torch
import so3_b200 as so3
busy = torch.empty(1 << 26, dtype=torch.float64).pin_memory()
sink = torch.empty_like(busy, device="cuda")
copies, side = torch.cuda.Stream(), torch.cuda.Stream()
ctx = so3.Context(0, stream=side)
for L in (367, 379, 439, 499):  # 2 L - 1: primes
    p = so3.SO3Parameters(L=L, N=2)
    x = torch.view_as_complex(torch.rand(so3.flmn_size(p), 2, dtype=torch.float64, device="cuda") - 0.5)
    out = [torch.empty(so3.f_size(p), dtype=torch.complex128, device="cuda") for _ in range(2)]
    back = [torch.zeros_like(x) for _ in range(2)]
    torch.cuda.synchronize()
    with torch.cuda.stream(copies):
        for _ in range(4):
            sink.copy_(busy, non_blocking=True)
    for i in range(2):
        ctx.inverse(x, p, out=out[i])
        ctx.forward(out[i], p, out=back[i])
        torch.cuda.synchronize()
    assert torch.isfinite(torch.view_as_real(out[0])).all()
    assert torch.equal(torch.view_as_real(out[0]), torch.view_as_real(out[1]))
    assert torch.equal(torch.view_as_real(back[0]), torch.view_as_real(back[1]))
"""


def test_first_calls_of_a_process():
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, env=dict(os.environ, PYTHONPATH=ROOT),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]

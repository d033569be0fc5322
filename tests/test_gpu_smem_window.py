"""Lengths whose DFT plans ask for just under 48 KB of dynamic shared memory:
with the kernels' static part that is more than a block gets without the
opt-in.  Each runs in a process of its own, where no earlier call has opted
in.  Against the oracle at the transform contract's 1e-12 (normwise)."""
import os
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import numpy as np
import so3_b200 as so3
from so3_b200 import synth
from oracle import oracle as O
from tests.helpers import oparams, params, rel_err
p = params({L}, {N}, sampling={sampling})
op = oparams(O, p)
fl = synth.gen_flmn(p, 4)
f = O.inverse(fl, op)
assert rel_err(so3.inverse(fl, p), f) < 1e-12
assert rel_err(so3.forward(f, p), O.forward(f, op)) < 1e-12
"""


@pytest.mark.parametrize("L,N,sampling", [(191, 2, 0), (255, 2, 0), (254, 2, 1)])
def test_first_call_of_a_process(O, L, N, sampling):
    r = subprocess.run([sys.executable, "-c", CODE.format(L=L, N=N, sampling=sampling)], cwd=ROOT,
                       env=dict(os.environ, PYTHONPATH=ROOT), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]

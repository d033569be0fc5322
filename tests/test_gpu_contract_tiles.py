"""The FP64 tensor-core contractions at the edges of their tiles (32 rows, 8 mu,
2 nu, 8 reduction entries) and of the Delta table's blocks of 8 degrees, odd
numbers of planes, L0 inside a block, real signals and their N = 1 case, more
planes than degrees, and |n| ranges that start between tiles (host buffers
staged in chunks): against the oracle, 1e-12 normwise (the transform
contract)."""
import numpy as np
import pytest

import so3_b200 as so3
from so3_b200 import synth
from tests.helpers import oparams, params, rel_err

TOL = 1e-12

pytestmark = pytest.mark.gpu

CASES = [dict(L=7, N=1), dict(L=8, N=2), dict(L=9, N=3, L0=5), dict(L=31, N=4, L0=9), dict(L=32, N=5),
         dict(L=33, N=6, storage=1), dict(L=40, N=7, mode=1), dict(L=41, N=2, mode=2), dict(L=3, N=5),
         dict(L=33, N=1, reality=1), dict(L=40, N=3, reality=1, storage=1), dict(L=65, N=9, method=1),
         dict(L=72, N=11, order=0, mode=3)]


@pytest.mark.parametrize("chunk", [None, "1"])
@pytest.mark.parametrize("kw", CASES, ids=lambda k: "-".join(f"{a}{b}" for a, b in k.items()))
def test_tile_edges_against_oracle(O, monkeypatch, kw, chunk):
    if chunk:  # every staged side splits into up to eight |n| ranges and row ranges
        monkeypatch.setenv("SO3GPU_STAGE_CHUNK_BYTES", chunk)
    p = params(**kw)
    op = oparams(O, p)
    fl = synth.gen_flmn(p, 23)
    f_ref = O.inverse(fl, op)
    assert rel_err(so3.inverse(fl, p), f_ref) < TOL
    rng = np.random.default_rng(7)
    f = rng.normal(size=f_ref.size)
    if not p.reality:
        f = f + 1j * rng.normal(size=f_ref.size)
    assert rel_err(so3.forward(f, p), O.forward(f, op)) < TOL
    assert so3.take_kernel_error() == 0

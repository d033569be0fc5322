"""The beta stages as matrix products at the edges of their tiles (16, 32 and 64
rows, 32 and 64 columns, 16 reduction entries; L + 1 rows on the MWSS grid) and
around the band limit where the inverse changes to DFTs: transforms against the
oracle, adjoints through <A x, y> = <x, A* y>.  Tolerance: the transform
contract's 1e-12 (normwise; inner products relative to the vectors' norms)."""
import numpy as np
import pytest

import so3_b200 as so3
from so3_b200 import synth
from tests.helpers import oparams, params, rel_err

TOL = 1e-12

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sampling", [0, 1])
@pytest.mark.parametrize("L", [1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 96, 97, 130])
def test_tile_edges_against_oracle(O, L, sampling):
    p = params(L, min(L, 3), sampling=sampling)
    op = oparams(O, p)
    fl = synth.gen_flmn(p, 5)
    f_ref = O.inverse(fl, op)
    assert rel_err(so3.inverse(fl, p), f_ref) < TOL
    # samples that are not band-limited exercise every entry of the matrices
    rng = np.random.default_rng(L)
    f = rng.normal(size=f_ref.size) + 1j * rng.normal(size=f_ref.size) if sampling == 0 else f_ref
    assert rel_err(so3.forward(f, p), O.forward(f, op)) < TOL


@pytest.mark.parametrize("L", [2, 17, 64, 97])
def test_adjoint_identities(L):
    p = params(L, 2)
    rng = np.random.default_rng(3 * L)
    x = synth.gen_flmn(p, 8)
    y = rng.normal(size=so3.f_size(p)) + 1j * rng.normal(size=so3.f_size(p))
    ax = so3.inverse(x, p)
    err = abs(np.vdot(ax, y) - np.vdot(x, so3.adjoint_inverse(y, p)))
    assert err < TOL * np.linalg.norm(ax) * np.linalg.norm(y)
    fy = so3.forward(y, p)
    err = abs(np.vdot(fy, x) - np.vdot(y, so3.adjoint_forward(x, p)))
    assert err < TOL * np.linalg.norm(fy) * np.linalg.norm(x)

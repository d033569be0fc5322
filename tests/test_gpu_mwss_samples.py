"""Forward transforms of MWSS samples that are no band-limited signal's: noise
reaches every entry of the analysis matrices, the rows b = 0 and b = L that mirror
onto themselves among them.  Against the oracle at the transform contract's 1e-12
(normwise)."""
import numpy as np
import pytest

import so3_b200 as so3
from tests.helpers import oparams, params, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", [0, 1])
@pytest.mark.parametrize("L", [1, 2, 3, 16, 33, 64, 100, 128])
def test_forward_of_noise(O, L, real):
    p = params(L, min(L, 3), sampling=1, reality=real)
    rng = np.random.default_rng(L)
    f = rng.normal(size=so3.f_size(p)) + (0 if real else 1j * rng.normal(size=so3.f_size(p)))
    assert rel_err(so3.forward(f, p), O.forward(f, oparams(O, p))) < 1e-12

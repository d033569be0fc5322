"""Gamma transforms too long for the one-level matrix tables (above 600 points:
N > 300, steerable signals likewise), which run on the scalar engines, and the
longest that still fit: both directions against the oracle.  1023 = 3 * 11 * 31
points (N = 512) has radices above 8 and, over alpha and beta, a compile-time
plan; 601 and 1021 are primes (Bluestein), 899 = 29 * 31.  Tolerance: the
transform contract's 1e-12 (normwise)."""
import numpy as np
import pytest

import so3_b200 as so3
from so3_b200 import synth
from tests.helpers import oparams, params, rel_err

TOL = 1e-12

pytestmark = pytest.mark.gpu

CASES = [(512, {}), (512, dict(reality=1)), (512, dict(sampling=1)), (511, {}), (450, {}), (450, dict(reality=1)),
         (301, {}), (300, {}), (300, dict(reality=1)), (256, dict(steerable=1)), (341, dict(steerable=1))]


@pytest.mark.parametrize("N,kw", CASES, ids=lambda v: str(v).replace(" ", ""))
def test_long_gamma_circles_against_oracle(O, N, kw):
    p = params(4, N, **kw)
    op = oparams(O, p)
    f_ref = O.inverse(synth.gen_flmn(p, N), op)
    assert rel_err(so3.inverse(synth.gen_flmn(p, N), p), f_ref) < TOL
    # samples of any gamma frequency: planes |n| >= L are not part of the band limit
    rng = np.random.default_rng(N)
    f = rng.normal(size=f_ref.size) + (0 if p.reality else 1j * rng.normal(size=f_ref.size))
    assert rel_err(so3.forward(f, p), O.forward(f, op)) < TOL


# the choice of engine by length and radices, on both sides of each line
CHOICE = [(49, n, {}) for n in (86, 88, 110, 113, 195, 199)] + [(49, n, dict(reality=1)) for n in (169, 172, 191, 200)] \
    + [(20, n, {}) for n in (50, 53)] + [(49, 90, dict(steerable=1))]


@pytest.mark.parametrize("L,N,kw", CHOICE, ids=lambda v: str(v).replace(" ", ""))
def test_either_engine_against_oracle(O, L, N, kw):
    p = params(L, N, **kw)
    op = oparams(O, p)
    fl = synth.gen_flmn(p, N)
    f_ref = O.inverse(fl, op)
    assert rel_err(so3.inverse(fl, p), f_ref) < TOL
    assert rel_err(so3.forward(f_ref, p), O.forward(f_ref, op)) < TOL

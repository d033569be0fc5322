"""The tensor-core DFT stages at the lengths where their plans can go wrong,
inverse and forward against the oracle: one level with and without the
separate sum (H a multiple of 8), two levels, Rader's and Bluestein's
convolutions, even lengths (MWSS, steerable gamma circles with a self-paired
entry), fewer columns than a task, and sequence counts that leave the last CTA
part empty.  Tolerance: the transform contract's 1e-12 (normwise)."""
import pytest

import so3_b200 as so3
from so3_b200 import synth
from tests.helpers import oparams, params, rel_err

TOL = 1e-12

pytestmark = pytest.mark.gpu

CASES = [
    # alpha / extended-beta length 2L-1 (MW) or 2L (MWSS)
    dict(L=9, N=2),                 # 17: one level, sum apart, one row tile
    dict(L=16, N=3),                # 31: one level, two full row tiles
    dict(L=17, N=4),                # 33: one level, sum apart
    dict(L=33, N=2, L0=2),          # 65
    dict(L=60, N=3),                # 119 = 17 * 7
    dict(L=63, N=2),                # 125 = 5^3
    dict(L=128, N=2),               # 255 = 17 * 15: both kinds of level
    dict(L=101, N=2),               # 201 = 67 * 3
    dict(L=300, N=1),               # 599: Rader over 598
    dict(L=234, N=2),               # 467: Bluestein (466 = 2 * 233)
    dict(L=32, N=3, sampling=1),    # 64
    dict(L=100, N=2, sampling=1),   # 200
    dict(L=251, N=1, sampling=1),   # 502 = 2 * 251
    # gamma length 2N-1, or 2N for steerable signals
    dict(L=12, N=1),
    dict(L=12, N=9),                # 17
    dict(L=40, N=33),               # 65
    dict(L=66, N=65),               # 129
    dict(L=12, N=8, steerable=1),   # 16
    dict(L=12, N=9, steerable=1),   # 18
    dict(L=40, N=33, steerable=1),  # 66
    dict(L=11, N=4, reality=1),
    dict(L=40, N=33, reality=1),
    dict(L=64, N=17, reality=1, sampling=1),
]


@pytest.mark.parametrize("kw", CASES, ids=lambda k: "-".join(f"{a}{b}" for a, b in k.items()))
def test_stage_lengths_against_oracle(O, kw):
    p = params(**kw)
    op = oparams(O, p)
    fl = synth.gen_flmn(p, 17)
    f_ref = O.inverse(fl, op)
    assert rel_err(so3.inverse(fl, p), f_ref) < TOL
    assert rel_err(so3.forward(f_ref, p), O.forward(f_ref, op)) < TOL

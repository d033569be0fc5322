"""Batches whose signals share stage launches, and the rule that sends parts of
split-precision batches to the FP64 contractions: FP64 batches longer than one
launch holds are bit-identical to single calls (same kernels, same arithmetic);
split batches and ragged calls with partly filled tiles stay within the split
path's 1e-10 of the FP64 path whichever contraction they take."""
import numpy as np
import pytest

import so3_b200 as so3
from so3_b200 import synth
from tests.helpers import params, rel_err

TOL_MIXED = 1e-10

pytestmark = pytest.mark.gpu


def _cpu(xs):
    import torch
    torch.cuda.synchronize()
    return [x.cpu().numpy() for x in xs]


@pytest.mark.parametrize("kw", [dict(L=17, N=5), dict(L=17, N=5, reality=1), dict(L=12, N=3, reality=1, sampling=1),
                                dict(L=20, N=4, steerable=1), dict(L=100, N=2), dict(L=9, N=1, reality=1)])
def test_fp64_batch_longer_than_a_launch(kw):
    import torch
    p = params(**kw)
    n = 35 if p.L < 50 else 5
    ctx = so3.Context(0)
    fls = [torch.from_numpy(synth.gen_flmn(p, 90 + i)).cuda() for i in range(n)]
    f = ctx.inverse_batch(fls, p, "fp64")
    b = ctx.forward_batch(f, p, "fp64")
    f, b = _cpu(f), _cpu(b)
    for i in range(n):
        one = ctx.inverse(fls[i], p)
        back = ctx.forward(one, p)
        one, back = _cpu([one, back])
        assert np.array_equal(f[i], one) and np.array_equal(b[i], back)


@pytest.mark.parametrize("kw", [dict(L=24, N=4, nsig=7), dict(L=24, N=4, nsig=11), dict(L=24, N=4, nsig=21),
                                dict(L=24, N=4, nsig=30), dict(L=33, N=3, nsig=18, reality=1),
                                dict(L=20, N=3, nsig=17, sampling=1)])
def test_split_batches_with_partly_filled_tiles(kw, monkeypatch):
    import torch
    monkeypatch.delenv("SO3GPU_DIGIT_TABLE", raising=False)
    kw = dict(kw)
    n = kw.pop("nsig")
    p = params(**kw)
    ctx = so3.Context(0)
    fls = [torch.from_numpy(synth.gen_flmn(p, 40 + i)).cuda() for i in range(n)]
    f64 = ctx.inverse_batch(fls, p, "fp64")
    b64 = _cpu(ctx.forward_batch(f64, p, "fp64"))
    fmx = _cpu(ctx.inverse_batch(fls, p, "mixed"))
    bmx = _cpu(ctx.forward_batch(f64, p, "mixed"))
    for x, y in list(zip(fmx, _cpu(f64))) + list(zip(bmx, b64)):
        assert rel_err(x, y) < TOL_MIXED
    assert so3.take_kernel_error() == 0


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("sizes", [[(24, 4)] * 13, [(24, 4)] * 3 + [(17, 2), (40, 6)], [(30, 3)] * 16 + [(8, 2)]])
def test_ragged_calls_on_either_path(sizes, pinned, monkeypatch):
    import torch
    if pinned:  # every tile on the split products
        monkeypatch.setenv("SO3GPU_DIGIT_TABLE", "0")
    else:
        monkeypatch.delenv("SO3GPU_DIGIT_TABLE", raising=False)
    ps = [params(L, N, method=i % 2) for i, (L, N) in enumerate(sizes)]
    ctx = so3.Context(0)
    fls = [torch.from_numpy(synth.gen_flmn(p, 7 + i)).cuda() for i, p in enumerate(ps)]
    f64 = [ctx.inverse(x, p) for x, p in zip(fls, ps)]
    b64 = _cpu([ctx.forward(x, p) for x, p in zip(f64, ps)])
    fmx = _cpu(ctx.inverse_ragged(fls, ps, "mixed"))
    bmx = _cpu(ctx.forward_ragged(f64, ps, "mixed"))
    for x, y in list(zip(fmx, _cpu(f64))) + list(zip(bmx, b64)):
        assert rel_err(x, y) < TOL_MIXED
    assert so3.take_kernel_error() == 0


def test_conv_batch_longer_than_a_launch():
    import torch
    p = params(16, 3)
    ctx = so3.Context(0)
    flm = torch.from_numpy(synth.gen_flm(16, 1)).cuda()
    glms = [torch.from_numpy(synth.gen_flm(16, 2 + i, mmax=2)).cuda() for i in range(34)]
    f = _cpu(ctx.s2toso3_inverse_batch(p, flm, glms, "fp64"))
    for i in (0, 31, 32, 33):
        assert np.array_equal(f[i], _cpu([ctx.inverse(ctx.s2toso3(p, flm, glms[i]), p)])[0])

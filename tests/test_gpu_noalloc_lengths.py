"""so3gpu_inverse_noalloc over the kinds of DFT plan that its static tables hold
(one and two matrix levels over alpha, one level or scalar passes over gamma),
in an order that changes one table at a time; bit for bit the allocating call."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
import so3_b200 as so3
from tests.helpers import params

pytestmark = pytest.mark.gpu

CASES = [dict(L=64, N=64), dict(L=64, N=64, order=0), dict(L=64, N=63), dict(L=63, N=63), dict(L=20, N=53),
         dict(L=20, N=64), dict(L=20, N=64, sampling=1), dict(L=64, N=64, sampling=1), dict(L=1, N=1), dict(L=2, N=1),
         dict(L=61, N=12, storage=1), dict(L=64, N=1)]


def test_lengths_in_turn():
    lib = so3._lib.load()
    stream = torch.cuda.current_stream()
    ctx = so3.Context(0, stream=stream)
    g = torch.Generator(device="cuda").manual_seed(3)
    for kw in CASES + CASES[::-1]:
        p = params(**kw)
        x = torch.rand(so3.flmn_size(p), 2, dtype=torch.float64, device="cuda", generator=g) - 0.5
        x = torch.view_as_complex(x)
        ref = ctx.inverse(x, p)
        out = torch.full_like(ref, float("nan"))
        q = p.to_struct()
        assert lib.so3gpu_inverse_noalloc(ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(x.data_ptr()),
                                          ctypes.byref(q), ctypes.c_void_p(stream.cuda_stream)) == 0, kw
        torch.cuda.synchronize()
        assert torch.equal(torch.view_as_real(out), torch.view_as_real(ref)), kw

"""MW alpha and beta circles whose length 2L - 1 is a prime and whose cyclic
convolution of length 2L - 2 splits into factors that need no padding: the
sequence buffers must still hold the 2L - 1 outputs and the 2L entries of a
column pair."""
import pytest

torch = pytest.importorskip("torch")
import so3_b200 as so3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [507, 367, 439])  # 1013 (46 x 22), 733, 877
@pytest.mark.parametrize("N", [1, 3])
def test_round_trip(L, N):
    p = so3.SO3Parameters(L=L, N=N)
    ctx = so3.Context(0)
    f = torch.empty(so3.f_size(p), dtype=torch.complex128, device="cuda")
    g = torch.Generator(device="cuda")
    g.manual_seed(L)
    x = torch.view_as_complex(torch.rand(so3.flmn_size(p), 2, dtype=torch.float64, device="cuda", generator=g) - 0.5)
    # entries with l < |n| are not part of the signal: one pass drops them
    y = torch.zeros_like(x)
    ctx.inverse(x, p, out=f)
    ctx.forward(f, p, out=y)
    z = torch.zeros_like(y)
    ctx.inverse(y, p, out=f)
    ctx.forward(f, p, out=z)
    assert y.abs().max() > 0.4
    assert (y - z).abs().max() <= 1e-11 * y.abs().max()

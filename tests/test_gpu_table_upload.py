"""First transforms of new lengths on streams that do not wait for the legacy
one: the DFT tables (index tables of Rader plans among them) must be complete
before a kernel reads them, also while large copies keep the copy engines busy."""
import pytest

torch = pytest.importorskip("torch")
import so3_b200 as so3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [367, 379, 439, 499])  # 2L - 1 = 733, 757, 877, 997: primes
def test_first_call_on_a_side_stream(L):
    p = so3.SO3Parameters(L=L, N=2)
    g = torch.Generator(device="cuda")
    g.manual_seed(L)
    fl = torch.view_as_complex(torch.rand(so3.flmn_size(p), 2, dtype=torch.float64, device="cuda", generator=g) - 0.5)
    first = torch.empty(so3.f_size(p), dtype=torch.complex128, device="cuda")
    again = torch.empty_like(first)
    busy = torch.empty(1 << 26, dtype=torch.float64).pin_memory()
    sink = torch.empty_like(busy, device="cuda")
    ctx = so3.Context(0)
    copies, side = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(copies):
        for _ in range(4):
            sink.copy_(busy, non_blocking=True)
    with torch.cuda.stream(side):
        ctx.inverse(fl, p, out=first)
    torch.cuda.synchronize()
    ctx.inverse(fl, p, out=again)
    torch.cuda.synchronize()
    assert torch.isfinite(torch.view_as_real(first)).all()
    assert torch.equal(torch.view_as_real(first), torch.view_as_real(again))

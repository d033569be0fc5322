"""A call that the device has no memory for is refused, and the next one runs."""
import pytest

torch = pytest.importorskip("torch")
import so3_b200 as so3
from tests.helpers import params

pytestmark = pytest.mark.gpu


def test_call_after_a_refused_allocation():
    big, small = params(512, 64), params(4, 512)
    fl = torch.empty(so3.flmn_size(big), dtype=torch.complex128, device="cuda")
    f = torch.empty(so3.f_size(big), dtype=torch.complex128, device="cuda")
    ctx = so3.Context(0)
    n = 96  # 290 GB of split-precision scratch; refused before any work on the buffers
    with pytest.raises(so3.SO3Error, match="status 4"):
        ctx.inverse_batch([fl] * n, big, "mixed", outs=[f] * n)
    x = torch.ones(so3.flmn_size(small), dtype=torch.complex128, device="cuda")
    y = ctx.inverse(x, small)  # the scalar gamma engine, which asks for launch errors
    torch.cuda.synchronize()
    assert torch.isfinite(torch.view_as_real(y)).all()

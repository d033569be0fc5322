"""CUDA graphs of transforms: what a context has to have built and kept for a
capture to work, and for its replay to stay valid."""
import pytest

torch = pytest.importorskip("torch")
import so3_b200 as so3
from tests.helpers import params

pytestmark = pytest.mark.gpu


def _coefficients(p, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand(so3.flmn_size(p), 2, dtype=torch.float64, device="cuda", generator=g) - 0.5
    return torch.view_as_complex(x)


def _samples(p):
    return torch.zeros(so3.f_size(p), dtype=torch.complex128, device="cuda")


@pytest.mark.parametrize("sampling", [0, 1])
def test_forward_captured_after_plain_inverse(sampling):
    p = params(83, 3, sampling=sampling)  # a band limit that no other test uses
    s = torch.cuda.Stream()
    ctx = so3.Context(0, stream=s)
    fl, f, back = _coefficients(p, 1), _samples(p), torch.zeros(so3.flmn_size(p), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    ctx.inverse(fl, p, out=f)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        ctx.forward(f, p, out=back)
    graph.replay()
    torch.cuda.synchronize()
    ref = ctx.forward(f, p)
    torch.cuda.synchronize()
    assert back.abs().max() > 0.1 and torch.equal(torch.view_as_real(back), torch.view_as_real(ref))


@pytest.mark.parametrize("prior", [0, 4])
def test_batches_beside_captured_transforms(prior):
    """After so3gpu_prepare single transforms and FP64 batches can be captured;
    uncaptured batches of more signals, before or after, take none of the
    scratch that the graphs hold."""
    p = params(24, 4)
    s = torch.cuda.Stream()
    ctx = so3.Context(0, stream=s)
    fls = [_coefficients(p, 10 + i) for i in range(33)]
    one, three = _samples(p), [_samples(p) for _ in range(3)]
    back = [torch.zeros_like(x) for x in fls[:3]]
    torch.cuda.synchronize()
    ctx.prepare(p)
    if prior:
        ctx.inverse_batch(fls[:prior], p, "fp64")
        torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        ctx.inverse(fls[0], p, out=one)
        ctx.inverse_batch(fls[1:4], p, "fp64", outs=three)
        ctx.forward_batch(three, p, "fp64", outs=back)
    f = ctx.inverse_batch(fls, p, "fp64")
    b = ctx.forward_batch(f, p, "fp64")
    torch.cuda.synchronize()
    for x in [one] + three + back:
        x.fill_(float("nan"))
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    for x, y in zip([one] + three + back, f[:4] + b[1:4]):
        assert torch.equal(torch.view_as_real(x), torch.view_as_real(y))

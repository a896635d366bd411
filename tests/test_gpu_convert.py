"""The conversions around the attention kernels for fp32 tensors against the same steps in torch: sizes around a vector and a
thread block, unaligned starts, infinities and NaN.  Powers of two and roundings are exact, so the bits are the same."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gen(n, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(n, generator=g, device="cuda") * scale


@pytest.mark.parametrize("sizes", [(1, 3, 5), (4096, 1023, 4), (1 << 20, 77777, 8)])
def test_abs_max(sizes):
    from kvax_b200.ops.flash_attention import _abs_max
    xs = [_gen(n, n) for n in sizes]
    assert torch.equal(_abs_max(*xs)[0], torch.stack([x.abs().amax() for x in xs]).max())
    xs[1] = _gen(sizes[1] + 1, 3)[1:]                                     # not on a 16-byte boundary
    xs[1][-1] = -1e30
    assert _abs_max(*xs).item() == torch.tensor(1e30).item()
    xs[2][0] = float("-inf")
    assert _abs_max(*xs).item() == float("inf")
    xs[0][0] = float("nan")
    assert torch.isnan(_abs_max(*xs)).item()
    assert _abs_max(xs[1].double(), xs[1][:0]).item() == torch.tensor(1e30).item()


@pytest.mark.parametrize("n", [1, 4, 1027, 1 << 18])
@pytest.mark.parametrize("scale", [1e-7, 1.0, 3e4])
def test_gradient_there_and_back(n, scale):
    from kvax_b200.ops.flash_attention import _FromOperand, _GradScaleBox, _ToOperand
    box = _GradScaleBox()
    x = torch.zeros(n, device="cuda", requires_grad=True)
    y = _FromOperand.apply(_ToOperand.apply(x, torch.float16, box), torch.float32, box)
    g = _gen(n, n, scale)
    (got,) = torch.autograd.grad(y, x, g)
    s = torch.exp2(-torch.floor(torch.log2(g.abs().amax().clamp_min(1e-30))))
    assert torch.equal(got, (g * s).to(torch.float16).to(torch.float32) * (1.0 / s))


def test_devices_must_agree():
    from kvax_b200 import _lib
    from kvax_b200.ops.flash_attention import _abs_max
    with pytest.raises(_lib.KvaxB200Error):
        _abs_max(torch.ones(4, device="cuda"), torch.ones(4))

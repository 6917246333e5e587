"""GPU tests of the one-launch gradient before the epilogue and of the operator's backward through it, against
the same expression in tensor operations: equal values (a NaN for a NaN), signs of zeros included."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def expression(gy, y, scale):
    g = gy.float()
    if y is not None:
        g = g * (y > 0)
    if scale is not None:
        g = g * scale
    return g.to(torch.bfloat16)


def same(a, b):
    nan = a.isnan() & b.isnan()
    return bool((nan | (a.view(torch.int16) == b.view(torch.int16))).all())


@pytest.mark.parametrize("kn,npix", [(8, 1), (8, 8192), (24, 8191), (136, 4000), (2048, 33)])
@pytest.mark.parametrize("relu", [True, False])
@pytest.mark.parametrize("scaled", [True, False])
def test_epilogue_grad_equals_the_expression(cglib, kn, npix, relu, scaled):
    from convgemm_gb300 import tc
    g = torch.Generator(device="cuda").manual_seed(kn + npix)
    bits = lambda: torch.randint(-32768, 32768, (npix, kn), device="cuda", generator=g).to(torch.int16).view(torch.bfloat16)  # noqa: E731
    gy, y = bits(), bits()   # every BF16 value: infinities, NaN, denormals, both zeros
    scale = torch.randn(kn, device="cuda", generator=g) if scaled else None
    dz = torch.full_like(gy, 7.0)
    tc.epilogue_grad_bf16(npix, kn, gy, y if relu else None, scale, dz)
    assert same(dz, expression(gy, y if relu else None, scale))


@pytest.mark.parametrize("scaled", [True, False])
@pytest.mark.parametrize("relu", [True, False])
@pytest.mark.parametrize("form", ["dense", "expanded", "transposed", "unaligned", "batched"])
def test_operator_backward_takes_every_gradient(cglib, form, relu, scaled):
    from convgemm_gb300 import torch_ops  # noqa: F401
    ops = torch.ops.convgemm
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(2, 9, 7, 16, device="cuda", generator=g).to(torch.bfloat16).requires_grad_()
    w = (torch.randn(16, 3, 3, 24, device="cuda", generator=g) * 0.1).requires_grad_()
    scale = torch.randn(24, device="cuda", generator=g) if scaled else None
    y = ops.conv2d_nhwc(x, w, scale, None, 1, 1, 1, relu)
    r = torch.randn(2 * 9 * 7 * 24 + 1, device="cuda", generator=g).to(torch.bfloat16)
    dense = r[:-1].view(2, 9, 7, 24)
    gy = {"dense": dense, "expanded": dense[:1, :1].expand(2, 9, 7, 24), "unaligned": r[1:].view(2, 9, 7, 24),
          "transposed": r[:-1].view(2, 7, 9, 24).transpose(1, 2), "batched": dense}[form]
    if form == "batched":
        got = torch.autograd.grad(y, (x, w), torch.stack([gy, -gy]), is_grads_batched=True)
        got = [t[0] for t in got]
    else:
        got = torch.autograd.grad(y, (x, w), gy)
    want = ops.conv2d_nhwc_backward(expression(gy, y.detach() if relu else None, scale), x.detach(), w.detach(), 1, 1, 1)
    cglib.check_device()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])

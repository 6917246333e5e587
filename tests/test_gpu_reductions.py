"""GPU tests of the one-launch reduction of many weight-gradient splits (groups of splits in order, then the groups)
and of the normalisation pass.

Weight gradients against FP64 convolutions of the same BF16 tensors, 1e-4 of the largest value (FP32 sums of at most
2704 products); the normalisation against FP64, 2^-8 of the value (one BF16 rounding, 2^-9, and an FP32 FMA)."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("layout", ["nhwc", "nchw"])
@pytest.mark.parametrize("x_on_a", [0, 0x10000])
@pytest.mark.parametrize("splits", [16, 17, 40, 169])
@pytest.mark.parametrize("c,kn,k", [(64, 64, 1), (72, 136, 1), (64, 200, 3), (128, 8, 3)])
def test_many_splits(cglib, c, kn, k, splits, x_on_a, layout):
    from convgemm_gb300 import tc
    cg = cglib
    b, hw = 16, 13
    s = cg.Shape.of(b, hw, hw, c, kn, k, k, k // 2, k // 2, 1, 1)
    g = torch.Generator(device="cuda").manual_seed(c + kn + splits)
    x = torch.randn(b, hw, hw, c, device="cuda", generator=g).to(torch.bfloat16)
    dy = torch.randn(b, hw, hw, kn, device="cuda", generator=g).to(torch.bfloat16)
    lay = cg.NHWC if layout == "nhwc" else cg.NCHW
    try:
        tc.tune_set(tc.TUNE_WGRAD, s, 64, splits | (x_on_a if kn >= 128 else 0))
        ws = torch.empty(tc.wgrad_bf16_workspace_size(s) // 4 + 4, device="cuda")
        dw = torch.full((c, k, k, kn) if layout == "nhwc" else (kn, c, k, k), float("nan"), device="cuda")
        tc.wgrad_bf16(lay, s, dy, x, dw, ws)
    finally:
        tc.tune_set(tc.TUNE_WGRAD, s, 0, 0)
    want = torch.nn.grad.conv2d_weight(x.double().permute(0, 3, 1, 2), (kn, c, k, k), dy.double().permute(0, 3, 1, 2),
                                       padding=k // 2)
    want = want.permute(1, 2, 3, 0) if layout == "nhwc" else want
    torch.cuda.synchronize()
    cg.check_device()
    assert ((dw.double() - want).abs().max() / want.abs().max()).item() <= 1e-4


@pytest.mark.parametrize("inplace", [False, True])
@pytest.mark.parametrize("npix,kn", [(1, 8), (999, 72), (4096, 64), (100000, 64), (1237, 200), (77, 2056), (3, 8200)])
def test_normalisation_pass(cglib, npix, kn, inplace):
    from convgemm_gb300 import tc
    g = torch.Generator(device="cuda").manual_seed(npix)
    z = torch.randn(npix, kn, device="cuda", generator=g).to(torch.bfloat16)
    scale, shift = torch.rand(kn, device="cuda", generator=g) + 0.5, torch.randn(kn, device="cuda", generator=g)
    a = z.double() * scale
    want = a + shift
    y = z.clone()
    tc.bn_apply_bf16(npix, kn, y if inplace else z, scale, shift, y, relu=False)
    # (FP32 rounding of the sum is relative to its terms)
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -22 * (a.abs() + shift.abs())).all()
    tc.bn_apply_bf16(npix, kn, z, scale, shift, y, relu=True)
    assert ((y.double() - want.clamp_min(0)).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -22 * (a.abs() + shift.abs())).all()

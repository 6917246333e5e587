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


@pytest.mark.parametrize("groups,kn", [(1, 64), (256, 16), (257, 16), (288, 128), (289, 128), (512, 72), (513, 72), (125, 512), (1024, 24),
                                       (1025, 24), (16384, 8), (16385, 8), (33300, 8)])
def test_statistics_and_column_sums_across_passes(cglib, groups, kn):
    """Batch statistics and the fused bias gradient where the reduction changes from one pass to two, and with fewer
    chunks of 256 groups than the second pass has rows, one more than it loads at once, and many. Operands with a mean, so
    that a lost chunk moves the sums by far more than the bound: FP32 accumulation of 16 products (2 * 16 roundings of
    2^-24 of their magnitudes) and of 32 rows (16 more), FP64 from there."""
    from convgemm_gb300 import tc
    cg = cglib
    P = 32 * groups - (groups % 7 if groups > 1 else 0)
    g = torch.Generator(device="cuda").manual_seed(groups + kn)
    s = cg.Shape.of(1, 1, P, 16, kn, 1, 1)
    x = torch.randn(P, 16, device="cuda", generator=g).add_(0.5).to(torch.bfloat16)
    w = torch.randn(16, kn, device="cuda", generator=g).add_(0.5).to(torch.bfloat16)
    wp = torch.empty(tc.weights_size(s, tc.OPERAND_FWD) // 2, dtype=torch.bfloat16, device="cuda")
    tc.pack_weights(cg.NHWC, s, tc.OPERAND_FWD, w.float(), wp)
    y = torch.empty(P, kn, dtype=torch.bfloat16, device="cuda")
    stats = torch.full((2, kn), float("nan"), dtype=torch.float64, device="cuda")
    for _ in range(2):
        tc.fwd_bf16_stats(s, x, wp, y, stats)
    z, m = x.double() @ w.double(), x.double().abs() @ w.double().abs()
    eps = 2.0 ** -24
    assert ((stats[0] - z.sum(0)).abs() <= 48 * eps * m.sum(0)).all()
    assert ((stats[1] - (z * z).sum(0)).abs() <= eps * (64 * (z.abs() * m).sum(0) + 16 * (z * z).sum(0))).all()

    # input gradient of a layer with `kn` input channels and 16 output channels
    d = cg.Shape.of(1, 1, P, kn, 16, 1, 1)
    dy, wt = x, w.t().contiguous()
    wpd = torch.empty(tc.weights_size(d, tc.OPERAND_DGRAD) // 2, dtype=torch.bfloat16, device="cuda")
    tc.pack_weights(cg.NHWC, d, tc.OPERAND_DGRAD, wt.float(), wpd)
    act = torch.randn(P, kn, device="cuda", generator=g).to(torch.bfloat16)
    dx, db = torch.empty_like(act), torch.full((kn,), float("nan"), device="cuda")
    for mask in (None, act):
        for _ in range(2):
            tc.dgrad_bf16_bias_grad(d, dy, wpd, dx, db, relu_x=mask)
        keep = 1.0 if mask is None else (act > 0).double()
        assert ((db.double() - (z * keep).sum(0)).abs() <= (48 + 1) * eps * (m * keep).sum(0)).all()
    torch.cuda.synchronize()
    cg.check_device()

"""GPU tests of output tiles that are not a power of two wide: the output channels are divided into equal
tiles of whole 16-column MMA widths, whose last 64-column chunk repeats columns of the chunk before (BF16
stores) and is cut to whole chunks where the output is accumulated.

Reference: FP64 convolutions of the same BF16 tensors.  BF16 outputs: one rounding (2^-9 of the value, two
where the output is accumulated) plus FP32 accumulation, 6e-3 of the largest value as for the other forms.
FP32 outputs of the 3xBF16 form: products to 2^-16, 1e-4 of the largest value."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

WIDTHS = [16, 48, 72, 80, 144, 192, 272, 400]


def nmax(got, want):
    return ((got.double() - want).abs().max() / want.abs().max()).item()


def tensors(cg, kn, stride, seed):
    s = cg.Shape.of(3, 15, 13, 64, kn, 3, 3, 1, 1, stride, stride)
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(3, 15, 13, 64, device="cuda", generator=g)
    wt = torch.randn(64, 3, 3, kn, device="cuda", generator=g) * (2 / 576) ** 0.5
    return s, x, wt, g


@pytest.mark.parametrize("bn", [0, 64, 128, 256])
@pytest.mark.parametrize("kn", WIDTHS)
def test_forward_widths(cglib, kn, bn):
    from convgemm_gb300 import tc
    cg = cglib
    s, x, wt, g = tensors(cg, kn, 1, kn)
    xb, wb = x.to(torch.bfloat16), wt.to(torch.bfloat16)
    z = torch.nn.functional.conv2d(xb.double().permute(0, 3, 1, 2), wb.double().permute(3, 0, 1, 2), padding=1)
    z = z.permute(0, 2, 3, 1)
    wp = torch.empty(tc.weights_size(s, tc.OPERAND_FWD) // 2, dtype=torch.bfloat16, device="cuda")
    tc.pack_weights(cg.NHWC, s, tc.OPERAND_FWD, wb.float(), wp)
    try:
        tc.tune_set(tc.TUNE_FWD, s, bn, 1 if bn else 0)
        y = torch.full((3, 15, 13, kn), float("nan"), dtype=torch.bfloat16, device="cuda")
        tc.fwd_bf16(s, xb, wp, y)
    finally:
        tc.tune_set(tc.TUNE_FWD, s, 0, 0)
    assert nmax(y, z) <= 6e-3

    # grouped: the same tiles; the packing of 64 channels is the same
    yg = torch.full_like(y, float("nan"))
    tc.Group([{"shape": s, "x": xb, "w": wp, "y": yg, "bn": bn}]).launch()
    assert nmax(yg, z) <= 6e-3

    # 3xBF16, FP32 output
    hi, lo = torch.empty_like(xb), torch.empty_like(xb)
    tc.split_bf16x2(x, hi, lo)
    wh, wl = torch.empty_like(wp), torch.empty_like(wp)
    tc.bf16x3_pack_weights(cg.NHWC, s, wt, wh, wl)
    y32 = torch.full((3, 15, 13, kn), float("nan"), device="cuda")
    tc.fwd_bf16x3(s, hi, lo, wh, wl, y32)
    z = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), wt.double().permute(3, 0, 1, 2), padding=1)
    torch.cuda.synchronize()
    cg.check_device()
    assert nmax(y32, z.permute(0, 2, 3, 1)) <= 1e-4


@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("c", [16, 72, 144, 272])
def test_input_gradient_widths(cglib, c, stride):
    from convgemm_gb300 import tc
    cg = cglib
    s = cg.Shape.of(3, 15, 13, c, 64, 3, 3, 1, 1, stride, stride)
    g = torch.Generator(device="cuda").manual_seed(c + stride)
    x = torch.randn(3, 15, 13, c, device="cuda", generator=g).to(torch.bfloat16)
    wt = (torch.randn(c, 3, 3, 64, device="cuda", generator=g) * (2 / 576) ** 0.5).to(torch.bfloat16).float()
    dy = torch.randn(3, s.ho, s.wo, 64, device="cuda", generator=g).to(torch.bfloat16)
    want = torch.nn.grad.conv2d_input((3, c, 15, 13), wt.double().permute(3, 0, 1, 2),
                                      dy.double().permute(0, 3, 1, 2), stride=stride, padding=1).permute(0, 2, 3, 1)
    wpd = torch.empty(tc.weights_size(s, tc.OPERAND_DGRAD) // 2, dtype=torch.bfloat16, device="cuda")
    tc.pack_weights(cg.NHWC, s, tc.OPERAND_DGRAD, wt, wpd)
    dx = torch.full_like(x, float("nan"))
    tc.dgrad_bf16(s, dy, wpd, dx)
    assert nmax(dx, want) <= 6e-3
    tc.dgrad_bf16_ex(s, dy, wpd, dx, accumulate=True)
    assert nmax(dx, 2 * want) <= 6e-3
    masked = torch.full_like(x, float("nan"))
    tc.dgrad_bf16_relu(s, dy, wpd, masked, x)
    torch.cuda.synchronize()
    cg.check_device()
    assert nmax(masked, torch.where(x > 0, want, torch.zeros_like(want))) <= 6e-3


def test_group_of_every_ring_class(cglib):
    """More tiles than CTAs in each class of widths (up to 64, 128, 256), long and short reductions, in one launch."""
    from convgemm_gb300 import tc
    cg = cglib
    g = torch.Generator(device="cuda").manual_seed(9)
    items, want = [], []
    for b, hw, c, kn, k in [(40, 28, 64, 48, 3), (64, 28, 40, 96, 1), (33, 27, 72, 144, 3), (90, 14, 128, 264, 1),
                            (64, 28, 24, 16, 1), (21, 30, 200, 128, 3), (2, 9, 8, 512, 5), (50, 28, 64, 64, 1)]:
        s = cg.Shape.of(b, hw, hw, c, kn, k, k, k // 2, k // 2, 1, 1)
        x = torch.randn(b, hw, hw, c, device="cuda", generator=g).to(torch.bfloat16)
        wt = (torch.randn(c, k, k, kn, device="cuda", generator=g) * (2 / (c * k * k)) ** 0.5).to(torch.bfloat16).float()
        wp = torch.empty(tc.group_weights_size(s) // 2, dtype=torch.bfloat16, device="cuda")
        tc.group_pack_weights(cg.NHWC, s, wt, wp)
        y = torch.full((b, hw, hw, kn), float("nan"), dtype=torch.bfloat16, device="cuda")
        items.append({"shape": s, "x": x, "w": wp, "y": y, "bn": 0})
        want.append(torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), wt.double().permute(3, 0, 1, 2),
                                               padding=k // 2).permute(0, 2, 3, 1))
    grp = tc.Group(items)
    for _ in range(2):
        grp.launch()
    torch.cuda.synchronize()
    cg.check_device()
    for it, z in zip(items, want):
        assert nmax(it["y"], z) <= 6e-3


@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("b,c", [(3, 64), (3, 72), (40, 72), (3, 144), (40, 144), (3, 272)])
def test_masked_input_gradient_in_place(cglib, b, c, stride):
    """dx == relu_x, widths that are and are not whole 64-column chunks, one to several tiles per CTA: the bits of the
    call with a separate dx, for the masked, the accumulating and the bias-gradient form."""
    from convgemm_gb300 import tc
    cg = cglib
    s = cg.Shape.of(b, 15, 13, c, 64, 3, 3, 1, 1, stride, stride)
    g = torch.Generator(device="cuda").manual_seed(c + stride)
    x = torch.randn(b, 15, 13, c, device="cuda", generator=g).to(torch.bfloat16)
    wt = torch.randn(c, 3, 3, 64, device="cuda", generator=g) * (2 / 576) ** 0.5
    dy = torch.randn(b, s.ho, s.wo, 64, device="cuda", generator=g).to(torch.bfloat16)
    wpd = torch.empty(tc.weights_size(s, tc.OPERAND_DGRAD) // 2, dtype=torch.bfloat16, device="cuda")
    tc.pack_weights(cg.NHWC, s, tc.OPERAND_DGRAD, wt, wpd)
    want, want_acc, db, db_in = torch.empty_like(x), x.clone(), torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
    tc.dgrad_bf16_bias_grad(s, dy, wpd, want, db, relu_x=x)
    tc.dgrad_bf16_ex(s, dy, wpd, want_acc, relu_x=x, accumulate=True)
    for _ in range(5):
        dx, dx_sum, dx_acc = x.clone(), x.clone(), x.clone()
        tc.dgrad_bf16_relu(s, dy, wpd, dx, dx)
        tc.dgrad_bf16_bias_grad(s, dy, wpd, dx_sum, db_in, relu_x=dx_sum)
        tc.dgrad_bf16_ex(s, dy, wpd, dx_acc, relu_x=dx_acc, accumulate=True)
        assert torch.equal(dx, want) and torch.equal(dx_sum, want) and torch.equal(dx_acc, want_acc)
        assert torch.equal(db_in, db)
    torch.cuda.synchronize()
    cg.check_device()

"""GPU tests of channel counts that are no multiple of 64: K blocks whose last channels the TMA loads
fill with zeros (forward, input gradient with one and with four stride-phase classes, weight gradient),
and the gathers that run where the blocks would be mostly padding.

Reference: FP64 convolutions of the same BF16 tensors.  BF16 outputs: one rounding (2^-9 of the value)
plus FP32 accumulation, 6e-3 of the largest value as for the other forms.  FP32 weight gradients: FP32
accumulation over at most 6272 pixels of products of unit-variance values, 1e-4 of the largest."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPES = [
    # b, h, w, c, kn, k, pad, stride, dil
    (2, 14, 13, 72, 136, 3, 1, 1, 1),     # second block: 8 of 64 channels
    (2, 15, 14, 136, 72, 3, 1, 2, 1),     # stride 2: four classes, tap counts 1 / 2 / 2 / 4
    (32, 14, 14, 120, 200, 3, 1, 1, 1),   # several tiles per CTA
    (3, 9, 11, 24, 312, 1, 0, 1, 1),      # one tap, one partial block
    (2, 12, 12, 88, 64, 5, 2, 1, 1),      # 25 taps
    (2, 13, 15, 40, 104, 3, 2, 1, 2),     # dilation 2
    (1, 9, 9, 16, 16, 3, 1, 2, 1),        # few channels: gathered
    (2, 10, 9, 8, 48, 3, 1, 1, 1),        # fewer still: no padding in the weight gradient either
]


def nmax(got, want):
    return ((got.double() - want).abs().max() / want.abs().max()).item()


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_ragged_channels_against_fp64(cglib, shape):
    from convgemm_gb300 import tc
    cg = cglib
    b, h, w, c, kn, k, pad, stride, dil = shape
    s = cg.Shape.of(b, h, w, c, kn, k, k, pad, pad, stride, stride, dil, dil)
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    x = torch.randn(b, h, w, c, device="cuda", generator=g).to(torch.bfloat16)
    wt = (torch.randn(c, k, k, kn, device="cuda", generator=g) * (2 / (c * k * k)) ** 0.5).to(torch.bfloat16).float()
    dy = torch.randn(b, s.ho, s.wo, kn, device="cuda", generator=g).to(torch.bfloat16)
    xd, wd, dyd = x.double().permute(0, 3, 1, 2), wt.double().permute(3, 0, 1, 2), dy.double().permute(0, 3, 1, 2)
    conf = dict(stride=stride, padding=pad, dilation=dil)

    wp = torch.empty(tc.weights_size(s, tc.OPERAND_FWD) // 2, dtype=torch.bfloat16, device="cuda")
    tc.pack_weights(cg.NHWC, s, tc.OPERAND_FWD, wt, wp)
    y, y2 = torch.empty_like(dy), torch.empty_like(dy)
    tc.fwd_bf16(s, x, wp, y)
    stats = torch.empty(2, kn, dtype=torch.float64, device="cuda")
    tc.fwd_bf16_stats(s, x, wp, y2, stats)
    z = torch.nn.functional.conv2d(xd, wd, **conf)
    assert nmax(y, z.permute(0, 2, 3, 1)) <= 6e-3
    assert torch.equal(y, y2)
    assert ((stats[0] - z.sum((0, 2, 3))).abs() <= 1e-4 * z.abs().sum((0, 2, 3))).all()

    wpd = torch.empty(tc.weights_size(s, tc.OPERAND_DGRAD) // 2, dtype=torch.bfloat16, device="cuda")
    tc.pack_weights(cg.NHWC, s, tc.OPERAND_DGRAD, wt, wpd)
    dx, dx2 = torch.empty_like(x), torch.empty_like(x)
    tc.dgrad_bf16(s, dy, wpd, dx)
    want = torch.nn.grad.conv2d_input(xd.shape, wd, dyd, **conf).permute(0, 2, 3, 1)
    assert nmax(dx, want) <= 6e-3
    tc.dgrad_bf16_relu(s, dy, wpd, dx2, x)
    assert torch.equal(dx2, torch.where(x > 0, dx, torch.zeros_like(dx)))
    db = torch.empty(c, device="cuda")
    tc.dgrad_bf16_bias_grad(s, dy, wpd, dx2, db, relu_x=x)
    masked = torch.where(x > 0, want, torch.zeros_like(want))
    assert torch.equal(dx2, torch.where(x > 0, dx, torch.zeros_like(dx)))
    assert ((db - masked.sum((0, 1, 2))).abs() <= 1e-4 * masked.abs().sum((0, 1, 2)) + 1e-6).all()

    ws = torch.empty(tc.wgrad_bf16_workspace_size(s) // 4 + 4, device="cuda")
    dw = torch.empty(c, k, k, kn, device="cuda")
    tc.wgrad_bf16(cg.NHWC, s, dy, x, dw, ws)
    want = torch.nn.grad.conv2d_weight(xd, wd.shape, dyd, **conf)
    assert nmax(dw, want.permute(1, 2, 3, 0)) <= 1e-4
    dwc = torch.empty(kn, c, k, k, device="cuda")
    tc.wgrad_bf16(cg.NCHW, s, dy, x, dwc, ws)
    torch.cuda.synchronize()
    cg.check_device()
    assert nmax(dwc, want) <= 1e-4


@pytest.mark.parametrize("shape,gathered", [
    ((64, 28, 28, 24, 384, 3, 1, 1, 1), True),     # dY on the 128-row side, 256 columns of taps and channels
    ((16, 56, 56, 40, 24, 5, 2, 1, 1), True),      # X on the 128-row side, 64 columns
    ((32, 28, 28, 104, 72, 3, 1, 2, 1), False),    # the same channels past 64, few pixels: by TMA
    ((4, 57, 55, 120, 128, 3, 1, 1, 1), False),    # the last of two boxes nearly full
], ids=str)
def test_weight_gradient_of_many_pixels(cglib, shape, gathered):
    """Both ways of loading ragged channels at the sizes where the estimates decide between them, with and without a tuning
    entry (which names tiles and splits, not the way). FP32 accumulation over at most 57600 pixels of unit-variance
    products: 1e-4 of the largest value."""
    from convgemm_gb300 import tc
    cg = cglib
    b, h, w, c, kn, k, pad, stride, dil = shape
    s = cg.Shape.of(b, h, w, c, kn, k, k, pad, pad, stride, stride, dil, dil)
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    x = torch.randn(b, h, w, c, device="cuda", generator=g).to(torch.bfloat16)
    dy = torch.randn(b, s.ho, s.wo, kn, device="cuda", generator=g).to(torch.bfloat16)
    want = torch.nn.grad.conv2d_weight(x.double().permute(0, 3, 1, 2), (kn, c, k, k), dy.double().permute(0, 3, 1, 2),
                                       stride=stride, padding=pad, dilation=dil)
    try:
        for bn, aux in ((0, 0), (128, 12 | tc.WGRAD_STAGES1)):
            tc.tune_set(tc.TUNE_WGRAD, s, bn, aux)
            if bn:   # ring stages: a flag of the TMA form, which the gathering one has not
                assert tc.tune_describe(tc.TUNE_WGRAD, s)[2] == (3 if gathered else 6)
            n = tc.wgrad_bf16_workspace_size(s)
            ws = torch.full((n // 4 + 4,), float("nan"), device="cuda")
            dw, dw2 = torch.empty(c, k, k, kn, device="cuda"), torch.empty(kn, c, k, k, device="cuda")
            tc.wgrad_bf16(cg.NHWC, s, dy, x, dw, ws)
            tc.wgrad_bf16(cg.NCHW, s, dy, x, dw2, ws)
            torch.cuda.synchronize()
            cg.check_device()
            assert nmax(dw, want.permute(1, 2, 3, 0)) <= 1e-4 and nmax(dw2, want) <= 1e-4
    finally:
        tc.tune_set(tc.TUNE_WGRAD, s, 0, 0)


@pytest.mark.parametrize("shape,gathered", [
    ((16, 28, 28, 40, 96, 3, 1, 1, 1), (True, False)),     # boxes off the 32-byte grid with a short tail
    ((16, 28, 28, 96, 40, 3, 1, 1, 1), (False, True)),     # the same for the input gradient's dY
    ((8, 31, 29, 32, 64, 7, 3, 1, 1), (False, False)),     # aligned rows, half a box
    ((4, 9, 7, 72, 32, 3, 1, 1, 1), (False, False)),       # few tiles
], ids=str)
def test_both_ways_of_loading_ragged_channels(cglib, shape, gathered):
    """Sizes on either side of the estimates' line, every form of each operation (equal bits) against FP64."""
    from convgemm_gb300 import tc
    b, h, w, c, kn, k, pad, stride, dil = shape
    s = cglib.Shape.of(b, h, w, c, kn, k, k, pad, pad, stride, stride, dil, dil)
    for op, by_threads in zip((tc.TUNE_FWD, tc.TUNE_DGRAD), gathered):
        _, bn, stages, _ = tc.tune_describe(op, s)
        assert (stages == {64: 8, 128: 6, 256: 4}[bn]) == by_threads, (op, bn, stages)   # the gathering ring
    test_ragged_channels_against_fp64(cglib, shape)

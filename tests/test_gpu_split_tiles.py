"""GPU tests of tiles whose K blocks a cluster of CTAs shares (launches of few tiles): forward with and without
statistics, masked, accumulating and bias-gradient input gradients (equal to one another bit by bit where they
compute the same sums), FP8 and 3xBF16; K blocks that do not divide evenly, stride-phase classes of different
lengths, channels that are no multiple of 64, ragged output widths.

Reference: FP64 convolutions of the same tensors, bounds as for the same forms without the split (BF16 outputs
6e-3 of the largest value, FP32 1e-4)."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPES = [
    # b, h, w, c, kn, k, stride
    (1, 14, 14, 256, 256, 3, 1),    # 36 blocks, 8 tiles
    (1, 7, 7, 512, 72, 3, 1),       # 72 blocks, a ragged second tile
    (2, 9, 11, 72, 136, 3, 1),      # zero-filled tails
    (1, 13, 13, 320, 40, 5, 1),     # 125 blocks
    (2, 15, 14, 256, 128, 3, 2),    # input gradient: four classes of 2, 4, 4, 8 blocks
    (1, 1, 1, 1024, 1000, 1, 1),    # one pixel
    (3, 14, 14, 192, 64, 3, 1),     # 27 blocks
]


def nmax(got, want):
    return ((got.double() - want).abs().max() / want.abs().max()).item()


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_split_tiles_against_fp64(cglib, shape):
    from convgemm_gb300 import tc
    cg = cglib
    b, h, w, c, kn, k, stride = shape
    s = cg.Shape.of(b, h, w, c, kn, k, k, k // 2, k // 2, stride, stride)
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    conf = dict(stride=stride, padding=k // 2)
    x32 = torch.randn(b, h, w, c, device="cuda", generator=g)
    w32 = torch.randn(c, k, k, kn, device="cuda", generator=g) * (2 / (c * k * k)) ** 0.5
    x, wt = x32.to(torch.bfloat16), w32.to(torch.bfloat16).float()
    dy = torch.randn(b, s.ho, s.wo, kn, device="cuda", generator=g).to(torch.bfloat16)
    scale, shift = torch.rand(kn, device="cuda", generator=g) + 0.5, torch.randn(kn, device="cuda", generator=g)
    xd, wd, dyd = x.double().permute(0, 3, 1, 2), wt.double().permute(3, 0, 1, 2), dy.double().permute(0, 3, 1, 2)
    z = torch.nn.functional.conv2d(xd, wd, **conf).permute(0, 2, 3, 1)

    wp = torch.empty(tc.weights_size(s, tc.OPERAND_FWD) // 2, dtype=torch.bfloat16, device="cuda")
    tc.pack_weights(cg.NHWC, s, tc.OPERAND_FWD, wt, wp)
    y, y2 = (torch.full((b, s.ho, s.wo, kn), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    tc.fwd_bf16(s, x, wp, y, scale, shift, relu=True)
    assert nmax(y, (z * scale + shift).clamp_min(0)) <= 6e-3
    stats = torch.empty(2, kn, dtype=torch.float64, device="cuda")
    tc.fwd_bf16(s, x, wp, y)
    for _ in range(3):
        tc.fwd_bf16_stats(s, x, wp, y2, stats)
    assert nmax(y, z) <= 6e-3 and torch.equal(y, y2)
    # FP32 accumulation errs by its products' magnitudes, not by the sum's: with one pixel a channel's sum may cancel
    # (at most 8000 products, a rounding of 2^-24 each, as a random walk 90 of them)
    mag = torch.nn.functional.conv2d(xd.abs(), wd.abs(), **conf).sum((0, 2, 3))
    assert ((stats[0] - z.sum((0, 1, 2))).abs() <= 90 * 2.0 ** -24 * mag).all()
    wpd = torch.empty(tc.weights_size(s, tc.OPERAND_DGRAD) // 2, dtype=torch.bfloat16, device="cuda")
    tc.pack_weights(cg.NHWC, s, tc.OPERAND_DGRAD, wt, wpd)
    want = torch.nn.grad.conv2d_input(xd.shape, wd, dyd, **conf).permute(0, 2, 3, 1)
    dx, dx2 = torch.full_like(x, float("nan")), torch.full_like(x, float("nan"))
    tc.dgrad_bf16(s, dy, wpd, dx)
    assert nmax(dx, want) <= 6e-3
    tc.dgrad_bf16_relu(s, dy, wpd, dx2, x)
    masked = torch.where(x > 0, dx, torch.zeros_like(dx))
    assert torch.equal(dx2, masked)
    db = torch.empty(c, device="cuda")
    tc.dgrad_bf16_bias_grad(s, dy, wpd, dx2, db, relu_x=x)
    wm = torch.where(x > 0, want, torch.zeros_like(want))
    magx = torch.nn.grad.conv2d_input(xd.shape, wd.abs(), dyd.abs(), **conf).sum((0, 2, 3))
    assert torch.equal(dx2, masked)
    assert ((db - wm.sum((0, 1, 2))).abs() <= 90 * 2.0 ** -24 * magx).all()
    tc.dgrad_bf16_ex(s, dy, wpd, dx, accumulate=True)
    assert nmax(dx, 2 * want) <= 6e-3

    if c % 64 == 0:
        z32 = torch.nn.functional.conv2d(x32.double().permute(0, 3, 1, 2), w32.double().permute(3, 0, 1, 2), **conf)
        hi, lo, wh, wl = torch.empty_like(x), torch.empty_like(x), torch.empty_like(wp), torch.empty_like(wp)
        tc.split_bf16x2(x32, hi, lo)
        tc.bf16x3_pack_weights(cg.NHWC, s, w32, wh, wl)
        y32 = torch.full((b, s.ho, s.wo, kn), float("nan"), device="cuda")
        tc.fwd_bf16x3(s, hi, lo, wh, wl, y32)
        assert nmax(y32, z32.permute(0, 2, 3, 1)) <= 1e-4
        q, qs = torch.empty(x.numel(), dtype=torch.uint8, device="cuda"), torch.empty(2, device="cuda")
        tc.fp8_quantize(x, q, qs)
        wq, ws = torch.empty(tc.fp8_weights_size(s), dtype=torch.uint8, device="cuda"), torch.empty(kn, device="cuda")
        tc.fp8_pack_weights(cg.NHWC, s, wt, wq, ws)
        o1, o2 = torch.empty(kn, device="cuda"), torch.empty(kn, device="cuda")
        tc.fp8_epilogue_scales(kn, None, None, ws, qs, o1, o2)
        tc.fwd_fp8(s, q, wq, y, o1, o2)
        # the quantised tensors themselves, multiplied in FP64
        xq = q.view(torch.float8_e4m3fn).double().view(b, h, w, c) * qs[0].double()
        wqd = (wt.double() / ws.double()).float().to(torch.float8_e4m3fn).double() * ws.double()
        zq = torch.nn.functional.conv2d(xq.permute(0, 3, 1, 2), wqd.permute(3, 0, 1, 2), **conf).permute(0, 2, 3, 1)
        assert nmax(y, zq) <= 6e-3
    torch.cuda.synchronize()
    cg.check_device()

"""GPU tests of the small-channel kernels (c <= 8): slabs of one column residue, shared by up to four output rows;
narrow and odd images, strides 1 to 3, dilation, several column chunks, an odd and an even number of taps.

Reference: FP64 convolutions of the same BF16 tensors, bounds as for the other BF16 forms (outputs 6e-3 of the
largest value, FP32 sums and weight gradients 1e-4)."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPES = [
    # b, h, w, c, kn, k, stride, pad, dil
    (2, 33, 47, 3, 64, 7, 2, 3, 1),
    (64, 30, 31, 3, 64, 7, 2, 3, 1),     # several groups of rows per CTA, ragged last group
    (1, 9, 1, 3, 64, 3, 2, 1, 1),        # no odd columns
    (2, 21, 22, 4, 96, 5, 3, 2, 1),
    (1, 40, 300, 1, 128, 3, 1, 1, 1),    # three column chunks
    (3, 17, 19, 8, 72, 3, 1, 2, 2),
    (16, 50, 18, 2, 64, 1, 1, 0, 1),     # one tap
    (4, 65, 63, 5, 64, 2, 2, 0, 1),      # an even number of taps
    (200, 7, 6, 3, 64, 3, 1, 1, 1),
]


def nmax(got, want):
    return ((got.double() - want).abs().max() / want.abs().max()).item()


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_small_channels_against_fp64(cglib, shape):
    from convgemm_gb300 import tc
    cg = cglib
    b, h, w, c, kn, k, stride, pad, dil = shape
    s = cg.Shape.of(b, h, w, c, kn, k, k, pad, pad, stride, stride, dil, dil)
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    x = torch.zeros(b, h, w, 8, dtype=torch.bfloat16, device="cuda")
    x[..., :c] = torch.randn(b, h, w, c, device="cuda", generator=g)
    wt = (torch.randn(c, k, k, kn, device="cuda", generator=g) * (2 / (c * k * k)) ** 0.5).to(torch.bfloat16).float()
    wp = torch.empty(tc.weights_size(s, tc.OPERAND_FWD) // 2, dtype=torch.bfloat16, device="cuda")
    tc.pack_weights(cg.NHWC, s, tc.OPERAND_FWD, wt, wp)
    conf = dict(stride=stride, padding=pad, dilation=dil)
    xd, wd = x[..., :c].double().permute(0, 3, 1, 2), wt.double().permute(3, 0, 1, 2)
    z = torch.nn.functional.conv2d(xd, wd, **conf).permute(0, 2, 3, 1)
    y, y2 = (torch.full((b, s.ho, s.wo, kn), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    stats = torch.empty(2, kn, dtype=torch.float64, device="cuda")
    tc.fwd_bf16(s, x, wp, y)
    tc.fwd_bf16_stats(s, x, wp, y2, stats)
    assert nmax(y, z) <= 6e-3 and torch.equal(y, y2)
    assert ((stats[0] - z.sum((0, 1, 2))).abs() <= 1e-4 * z.abs().sum((0, 1, 2))).all()
    assert ((stats[1] - (z * z).sum((0, 1, 2))).abs() <= 1e-4 * (z * z).sum((0, 1, 2))).all()

    # an infinity reaches the outputs whose windows hold it and no others
    hit = torch.zeros_like(xd[:, :1])
    hit[b // 2, 0, h // 2, w // 2] = 1
    x[b // 2, h // 2, w // 2, 0] = float("inf")
    tc.fwd_bf16(s, x, wp, y2)
    near = torch.nn.functional.conv2d(hit, torch.ones_like(wd[:1, :1]), **conf)[:, 0] > 0
    assert torch.equal(y2[~near], y[~near]) and not y2[near].isfinite().any()
    x[b // 2, h // 2, w // 2, 0] = 0

    dy = torch.randn(b, s.ho, s.wo, kn, device="cuda", generator=g).to(torch.bfloat16)
    ws = torch.empty(tc.wgrad_bf16_workspace_size(s) // 4 + 4, device="cuda")
    dw = torch.empty(c, k, k, kn, device="cuda")
    tc.wgrad_bf16(cg.NHWC, s, dy, x, dw, ws)
    want = torch.nn.grad.conv2d_weight(x[..., :c].double().permute(0, 3, 1, 2), wd.shape,
                                       dy.double().permute(0, 3, 1, 2), **conf)
    torch.cuda.synchronize()
    cg.check_device()
    assert nmax(dw, want.permute(1, 2, 3, 0)) <= 1e-4

"""GPU tests of the preparation and reduction kernels at the sizes where their vector, tile and
remainder paths begin and end: casts and splits are exact element by element (compared bit for bit
with PyTorch), packings equal the per-layer kernels' bits, column sums stay within FP32 rounding of
an FP64 sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def offset(t, off):
    """A copy of t whose first element sits `off` elements into its allocation."""
    buf = torch.empty(t.numel() + off, dtype=t.dtype, device=t.device)
    buf[off:] = t.reshape(-1)
    return buf[off:]


@pytest.mark.parametrize("nchw", [True, False])
@pytest.mark.parametrize("b,c,h,w", [(2, 3, 9, 7), (1, 8, 16, 16), (3, 9, 8, 8), (2, 64, 8, 8), (2, 65, 7, 9), (1, 136, 5, 13)])
@pytest.mark.parametrize("off_in,off_out", [(0, 0), (1, 0), (0, 1)])
def test_cast_to_bf16_nhwc(cglib, nchw, b, c, h, w, off_in, off_out):
    from convgemm_gb300 import tc
    g = torch.Generator(device="cuda").manual_seed(c)
    x = torch.randn(b, c, h, w, device="cuda", generator=g)
    src = x if nchw else x.permute(0, 2, 3, 1).contiguous()
    out = offset(torch.full((b, h, w, tc.c8(c)), 7.0, dtype=torch.bfloat16, device="cuda"), off_out)
    tc.to_bf16_nhwc(cglib.NCHW if nchw else cglib.NHWC, b, c, h, w, offset(src, off_in), out)
    got = out.view(b, h, w, tc.c8(c))
    assert torch.equal(got[..., :c], x.permute(0, 2, 3, 1).to(torch.bfloat16))
    assert not got[..., c:].any()


@pytest.mark.parametrize("n,off", [(1, 0), (7, 0), (8, 0), (4099, 0), (4096, 1), (1245184 + 5, 0)])
@pytest.mark.parametrize("bf16", [True, False])
def test_quantize_and_split(cglib, n, off, bf16):
    from convgemm_gb300 import tc
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, device="cuda", generator=g)
    xs = offset(x.to(torch.bfloat16) if bf16 else x, off)
    q, scale = torch.empty(n, dtype=torch.uint8, device="cuda"), torch.empty(2, device="cuda")
    tc.fp8_quantize(xs, q, scale)
    xf = xs.float()
    sc = np.float32(xf.abs().max().item()) / np.float32(448)   # IEEE division (a CUDA tensor / scalar is a multiplication)
    assert scale[0].item() == sc
    want = (xf * float(np.float32(1) / sc)).clamp(-448, 448).to(torch.float8_e4m3fn)
    assert torch.equal(q, want.view(torch.uint8))
    if not bf16:
        hi, lo = (torch.empty(n, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        tc.split_bf16x2(xs, hi, lo)
        assert torch.equal(hi, x.to(torch.bfloat16))
        assert torch.equal(lo, (x - hi.float()).to(torch.bfloat16))


@pytest.mark.parametrize("c,kn,k,stride", [(3, 8, 7, 2), (8, 65, 1, 1), (70, 40, 3, 2), (520, 24, 3, 1), (24, 136, 5, 1)])
def test_grouped_nchw_packing_matches_single(cglib, c, kn, k, stride):
    from convgemm_gb300 import tc
    s = cglib.Shape.of(2, 12, 12, c, kn, k, k, k // 2, k // 2, stride, stride)
    w = torch.randn(kn, c, k, k, device="cuda")
    one, two = [], []
    for op in (tc.OPERAND_FWD, tc.OPERAND_DGRAD):
        n = tc.weights_size(s, op) // 2
        one.append(torch.full((n,), 3.0, dtype=torch.bfloat16, device="cuda"))
        two.append(torch.full((n,), 5.0, dtype=torch.bfloat16, device="cuda"))
        tc.pack_weights(cglib.NCHW, s, op, w, one[-1])
    tc.Prep([dict(layout=cglib.NCHW, shape=s, weights=w, packed_fwd=two[0], packed_dgrad=two[1])]).launch()
    torch.cuda.synchronize()
    assert torch.equal(one[0], two[0]) and torch.equal(one[1], two[1])


@pytest.mark.parametrize("b,h,w,c,kn", [(1, 1, 31, 64, 72), (2, 40, 26, 64, 8), (2, 255, 260, 8, 72)])
def test_column_sums(cglib, b, h, w, c, kn):
    """Bias gradient and fused bias gradient below, at and above one chunk of statistics groups (65
    groups: two chunks; 4144: the second pass's batched loads).  FP32 sums of n terms stay within
    n_rows * 2^-24 of the sum of magnitudes, with at most 256 terms in a row before they are added up."""
    from convgemm_gb300 import tc
    s = cglib.Shape.of(b, h, w, c, kn, 1, 1)
    g = torch.Generator(device="cuda").manual_seed(h)
    dy = torch.randn(b, h, w, kn, device="cuda", generator=g).to(torch.bfloat16)
    tol = 600 * 2.0 ** -24
    db = torch.empty(kn, device="cuda")
    for t in (dy, offset(dy, 1)):
        tc.bias_grad_bf16(s, t, db)
        ref = dy.double().sum((0, 1, 2))
        assert ((db.double() - ref).abs() <= tol * dy.double().abs().sum((0, 1, 2))).all()
    wt = torch.randn(c, 1, 1, kn, device="cuda", generator=g)
    wp = torch.empty(tc.weights_size(s, tc.OPERAND_DGRAD) // 2, dtype=torch.bfloat16, device="cuda")
    tc.pack_weights(cglib.NHWC, s, tc.OPERAND_DGRAD, wt, wp)
    x = torch.randn(b, h, w, c, device="cuda", generator=g).to(torch.bfloat16)
    dx, dx2 = torch.empty_like(x), torch.empty_like(x)
    dbx = torch.empty(c, device="cuda")
    tc.dgrad_bf16_bias_grad(s, dy, wp, dx, dbx, relu_x=x)
    tc.dgrad_bf16_relu(s, dy, wp, dx2, x)
    torch.cuda.synchronize()
    cglib.check_device()
    assert torch.equal(dx, dx2)
    # the sums are of the FP32 accumulators, dx of their BF16 rounding: 2^-8 of each term
    ref = dx.double().sum((0, 1, 2))
    assert ((dbx.double() - ref).abs() <= (2.0 ** -8 + tol) * dx.double().abs().sum((0, 1, 2))).all()


@pytest.mark.parametrize("b,c,h,w", [(3, 3, 33, 31), (2, 1, 32, 32), (2, 8, 41, 25), (5, 4, 64, 64), (1, 7, 129, 127)])
def test_few_channel_cast_blocks_of_pixels(cglib, b, c, h, w):
    """NCHW with c <= 8: 1024 pixels of an image per block (1023 to 16383 pixels), the values rounded as by torch."""
    from convgemm_gb300 import tc
    x = torch.randn(b, c, h, w, device="cuda")
    out = torch.full((b, h, w, 8), float("nan"), dtype=torch.bfloat16, device="cuda")
    tc.to_bf16_nhwc(cglib.NCHW, b, c, h, w, x, out)
    want = torch.zeros_like(out)
    want[..., :c] = x.permute(0, 2, 3, 1).to(torch.bfloat16)
    assert torch.equal(out, want)


@pytest.mark.parametrize("b,h,w,kn", [(1, 1, 1, 8), (1, 1, 129, 72), (1, 1, 1025, 64), (1, 45, 46, 136), (2, 420, 317, 24)])
@pytest.mark.parametrize("off", [0, 1])
def test_bias_gradient_groups(cglib, b, h, w, kn, off):
    """One pixel, one more than a block's rows, one more than a group, ragged groups, groups of more than 1024 pixels. Of a
    sum of n terms in groups of at most 1041 pixels, each term passes at most 9 + 8 + 16 + 256 FP32 additions."""
    from convgemm_gb300 import tc
    s = cglib.Shape.of(b, h, w, 64, kn, 1, 1)
    g = torch.Generator(device="cuda").manual_seed(w)
    dy = torch.randn(b, h, w, kn, device="cuda", generator=g).add_(0.25).to(torch.bfloat16)
    db, db2 = (torch.full((kn,), float("nan"), device="cuda") for _ in range(2))
    tc.bias_grad_bf16(s, offset(dy, off), db)
    tc.bias_grad_bf16(s, offset(dy, off), db2)
    ref, mag = dy.double().sum((0, 1, 2)), dy.double().abs().sum((0, 1, 2))
    assert torch.equal(db, db2)
    assert ((db.double() - ref).abs() <= 289 * 2.0 ** -24 * mag).all()

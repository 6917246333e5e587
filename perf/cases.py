"""Performance cases of convgemm_gb300: the calls a user's program makes, through the public entry points.

A case is a dict of plain values; its "kind" names the call pattern:

infer       one BF16 inference layer: folded batch norm + ReLU, weights packed once and kept
block       one training step of a bottleneck block (1x1, 3x3, 1x1, bias + ReLU) in BF16: the FP32 master
            weights packed, three forwards, three input gradients (the inner two with the ReLU mask and the
            previous layer's bias gradient fused) and three weight gradients
stem        the first layer in training: FP32 NCHW images converted, weights packed, forward with batch
            statistics, batch-norm fold and apply, weight gradient
nchw        one training layer on NCHW FP32 tensors in BF16: both tensors converted, weights packed, forward,
            input gradient, weight gradient in the NCHW API's layout, bias gradient
fp8         one FP8-E4M3 inference layer: the BF16 activation quantised, scales folded, forward
bf16x3      one 3xBF16 inference layer: the FP32 activation split, forward with FP32 output
group       many BF16 convolutions of uneven shapes in one persistent launch
torch       the PyTorch operator with autograd: forward, input gradient, weight gradient
f32_host    the FP32 drop-in on host arrays, as a ctypes caller of the reference makes it (forward, bias + ReLU)
f32         one FP32 training layer on the GPU: forward with bias + ReLU, input gradient, weight gradient

Activations are what a ReLU leaves of N(0, 1), images N(0, 1), weights Kaiming-normal, gradients N(0, 1e-2).
The library's own tile choices are used: no tuning table is loaded.
"""
import math

import numpy as np
import torch

import convgemm_gb300 as cg
from convgemm_gb300 import tc, torch_ops, workloads  # noqa: F401  (torch_ops registers the operator)

BF16, F32 = torch.bfloat16, torch.float32


def listed():
    return [
        # one image, one ResNet stage-3 layer: serving at batch 1, where latency and launches count
        dict(name="infer_b1_14x14_256", kind="infer", b=1, h=14, w=14, c=256, kn=256, k=3, stride=1),
        # ResNet-50 training, batch 64: an identity block of the first stage (large pixels, few channels) ...
        dict(name="block_56x56_64", kind="block", b=64, h=56, w=56, c=256, mid=64, kn=256, stride=1),
        # ... and one of the third stage (few pixels, many channels), the most frequent block of the network
        dict(name="block_14x14_256", kind="block", b=64, h=14, w=14, c=1024, mid=256, kn=1024, stride=1),
        # the ResNet-50 stem, batch 64, with training-mode batch norm
        dict(name="stem_224x224", kind="stem", b=64, h=224, w=224, c=3, kn=64, k=7, stride=2),
        # a VGG-16 layer of an NCHW program, batch 32
        dict(name="nchw_28x28_512", kind="nchw", b=32, h=28, w=28, c=512, kn=512, k=3),
        # the precision forms on ResNet-50 layers, batch 128
        dict(name="fp8_28x28_128", kind="fp8", b=128, h=28, w=28, c=128, kn=128, k=3, stride=1),
        dict(name="bf16x3_14x14_256", kind="bf16x3", b=128, h=14, w=14, c=256, kn=256, k=3, stride=1),
        # a quarter of the 256 uneven convolutions of the grouped workload
        dict(name="group_64", kind="group", n=64, shapes=2024),
        # a strided layer of odd sizes and channels in a PyTorch training loop
        dict(name="torch_37x45_72", kind="torch", b=12, h=37, w=45, c=72, kn=136, k=3, stride=2, dil=1),
        # the drop-in as the reference's callers use it: host arrays, batch 8
        dict(name="f32_host_28x28_64", kind="f32_host", b=8, h=28, w=28, c=64, kn=64, k=3),
        # FP32 training on the GPU: a strided ResNet-50 layer (NHWC) and a VGG-16 layer (NCHW)
        dict(name="f32_nhwc_56x56_128_s2", kind="f32", layout="nhwc", b=64, h=56, w=56, c=128, kn=128, k=3, stride=2),
        dict(name="f32_nchw_56x56_256", kind="f32", layout="nchw", b=32, h=56, w=56, c=256, kn=256, k=3, stride=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _chan(rng, lo, hi, step):
    return max(step, _log(rng, lo, hi) // step * step)


def _draw(rng):
    kind = rng.choice(["infer", "block", "stem", "nchw", "fp8", "bf16x3", "group", "torch", "f32_host", "f32", "f32"])
    h = _log(rng, 7, 112)
    w = max(5, h + rng.choice([0, 0, 0, -1, 3, 9]))
    k = rng.choice([1, 3, 3, 5])
    st = rng.choice([1, 1, 2])
    step = rng.choice([8, 16, 64])
    if kind == "group":
        return dict(kind=kind, n=rng.randint(8, 64), shapes=rng.randint(1, 1 << 20))
    if kind == "infer":
        return dict(kind=kind, b=_log(rng, 1, 8), h=h, w=w, c=_chan(rng, 16, 1024, step), kn=_chan(rng, 16, 1024, step),
                    k=k, stride=st)
    if kind == "block":
        mid = _chan(rng, 32, 512, step)
        return dict(kind=kind, b=_log(rng, 4, 64), h=h, w=w, c=_chan(rng, 64, 1024, step), mid=mid, kn=4 * mid, stride=st)
    if kind == "stem":
        h = _log(rng, 32, 256)
        return dict(kind=kind, b=_log(rng, 4, 64), h=h, w=h + rng.choice([0, 0, 1, 8]), c=rng.choice([1, 3, 3, 4]),
                    kn=rng.choice([32, 48, 64, 64, 96]), k=rng.choice([3, 5, 7]), stride=rng.choice([1, 2, 2]))
    if kind == "nchw":
        return dict(kind=kind, b=_log(rng, 2, 64), h=h, w=w, c=_chan(rng, 32, 512, step), kn=_chan(rng, 32, 512, step),
                    k=rng.choice([1, 3, 3]))
    if kind in ("fp8", "bf16x3"):
        return dict(kind=kind, b=_log(rng, 1, 128), h=h, w=w, c=_chan(rng, 64, 1024, 64), kn=_chan(rng, 32, 1024, step),
                    k=k, stride=st)
    if kind == "torch":
        return dict(kind=kind, b=_log(rng, 1, 64), h=h, w=w, c=_chan(rng, 16, 512, 8), kn=_chan(rng, 16, 512, 8), k=k,
                    stride=st, dil=rng.choice([1, 1, 2]) if k > 1 and h > 10 else 1)
    if kind == "f32_host":
        return dict(kind=kind, b=_log(rng, 1, 16), h=h, w=w, c=_log(rng, 3, 256), kn=_log(rng, 8, 256), k=k)
    return dict(kind=kind, layout=rng.choice(["nhwc", "nchw"]), b=_log(rng, 1, 64), h=h, w=w, c=_log(rng, 3, 512),
                kn=_log(rng, 8, 512), k=k, stride=st)


def draw(rng):
    # no drawn case costs more than the largest listed one (the FP32 VGG-16 layer)
    most = {"f32": 250e9, "f32_host": 10e9, "infer": 100e9}
    while True:
        c = _draw(rng)
        w = work(c)
        if w["flops"] <= most.get(c["kind"], 1000e9 if c["kind"] != "group" else 2500e9) and w["bytes"] <= 2e9:
            return c


# ------------------------------------------------------------------ geometry
def _shape(case, c=None, kn=None, k=None, stride=None, hw=None):
    c, kn = c or case["c"], kn or case["kn"]
    k, stride = k or case["k"], stride or case.get("stride", 1)
    h, w = hw or (case["h"], case["w"])
    dil = case.get("dil", 1)
    pad = dil * (k - 1) // 2
    return cg.Shape.of(case["b"], h, w, c, kn, k, k, pad, pad, stride, stride, dil, dil)


def _block_shapes(case):
    s2 = _shape(case, case["mid"], case["mid"], 3)
    return [_shape(case, case["c"], case["mid"], 1, 1), s2,
            _shape(case, case["mid"], case["kn"], 1, 1, (s2.ho, s2.wo))]


def _flops(s):
    return 2 * s.b * s.ho * s.wo * s.kn * s.c * s.kh * s.kw


def _group_convs(case):
    return workloads.uneven_convs(case["n"], case["shapes"])


def _group_shape(d):
    return cg.Shape.of(d["b"], d["h"], d["w"], d["c"], d["kn"], d["k"], d["k"], d["pad"], d["pad"], d["stride"], d["stride"])


def work(case):
    kind = case["kind"]
    if kind == "block":
        s = _block_shapes(case)
        px, py, pm = (s[0].b * a * b for a, b in ((s[0].h, s[0].w), (s[2].ho, s[2].wo), (s[0].ho, s[0].wo)))
        wts = sum(t.c * t.kh * t.kw * t.kn for t in s)
        act = 2 * px * s[0].c + 2 * py * s[2].kn + pm * s[0].kn + py * s[1].kn   # x, dx; y, dy; the inner gradients
        return {"bytes": 2 * act + 2 * 4 * wts, "flops": 3 * sum(_flops(t) for t in s)}
    if kind == "group":
        shapes = [_group_shape(d) for d in _group_convs(case)]
        return {"bytes": sum(2 * (s.b * s.h * s.w * s.c + s.c * s.kh * s.kw * s.kn + s.b * s.ho * s.wo * s.kn) for s in shapes),
                "flops": sum(_flops(s) for s in shapes)}
    s = _shape(case)
    x, y, wt = s.b * s.h * s.w * s.c, s.b * s.ho * s.wo * s.kn, s.c * s.kh * s.kw * s.kn
    nbytes, passes = {
        "infer": (2 * (x + y + wt), 1), "stem": (4 * x + 2 * 2 * y + 2 * 4 * wt, 2),
        "nchw": (4 * x + 4 * y + 2 * x + 2 * y + 2 * 4 * wt, 3), "fp8": (2 * x + 2 * y + wt, 1),
        "bf16x3": (4 * x + 4 * y + 4 * wt, 1), "torch": (2 * 2 * (x + y) + 2 * 4 * wt, 3),
        "f32_host": (4 * (x + y + wt), 1), "f32": (2 * 4 * (x + y + wt), 3)}[kind]
    return {"bytes": nbytes, "flops": passes * _flops(s)}


# -------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, std=1.0):
    return torch.randn(*shape, device="cuda", generator=g).mul_(std)


def _weights(g, s, nchw=False):
    shape = (s.kn, s.c, s.kh, s.kw) if nchw else (s.c, s.kh, s.kw, s.kn)
    return _randn(g, *shape, std=math.sqrt(2 / (s.c * s.kh * s.kw)))


def _act(g, *shape):
    return _randn(g, *shape).relu_()


def _uniform(g, n, lo, hi):
    return torch.rand(n, device="cuda", generator=g).mul_(hi - lo).add_(lo)


def _bn(g, kn):
    return dict(mean=_randn(g, kn, std=0.1), inv_std=1 / _uniform(g, kn, 0.5, 2).sqrt(), gamma=_uniform(g, kn, 0.5, 1.5),
                beta=_uniform(g, kn, -0.1, 0.1))


def _inputs(case, seed):
    """The tensors a program has before the call, from the seed alone."""
    kind = case["kind"]
    if kind == "f32_host":
        r, s = np.random.default_rng(seed), _shape(case)
        return dict(x=r.uniform(-1, 1, (s.b, s.h, s.w, s.c)).astype(np.float32),
                    w=(r.standard_normal((s.c, s.kh, s.kw, s.kn)) * math.sqrt(2 / (s.c * s.kh * s.kw))).astype(np.float32),
                    bias=r.uniform(-0.1, 0.1, s.kn).astype(np.float32))
    g = _gen(seed)
    if kind == "block":
        s = _block_shapes(case)
        return dict(x=_act(g, s[0].b, s[0].h, s[0].w, s[0].c).to(BF16), w=[_weights(g, t) for t in s],
                    bias=[_uniform(g, t.kn, -0.1, 0.1) for t in s],
                    dy=_randn(g, s[2].b, s[2].ho, s[2].wo, s[2].kn, std=1e-2).to(BF16))
    if kind == "group":
        out = []
        for d in _group_convs(case):
            s = _group_shape(d)
            out.append(dict(x=torch.rand(s.b, s.h, s.w, s.c, device="cuda", generator=g).mul_(2).sub_(1).to(BF16),
                            w=_weights(g, s), bias=_uniform(g, s.kn, -0.1, 0.1)))
        return out
    s = _shape(case)
    nchw = kind in ("nchw", "stem") or case.get("layout") == "nchw"
    i = dict(w=_weights(g, s, nchw and kind != "stem"))
    xs = (s.b, s.c, s.h, s.w) if nchw else (s.b, s.h, s.w, s.c)
    ys = (s.b, s.kn, s.ho, s.wo) if nchw and kind != "stem" else (s.b, s.ho, s.wo, s.kn)
    i["x"] = _randn(g, *xs) if kind == "stem" else _act(g, *xs)
    i["bias"] = _uniform(g, s.kn, -0.1, 0.1)
    if kind in ("infer", "fp8", "bf16x3", "stem"):
        i.update(_bn(g, s.kn))
    if kind in ("stem", "nchw", "torch", "f32"):
        i["dy"] = _randn(g, *ys, std=1e-2)
    if kind in ("infer", "fp8", "torch"):
        i["x"] = i["x"].to(BF16)
    if kind in ("stem", "torch"):
        i["dy"] = i["dy"].to(BF16)
    return i


def _empty(*shape, dtype=BF16):
    return torch.empty(*shape, dtype=dtype, device="cuda")


def _packed(s, kind):
    return _empty(max(64, tc.weights_size(s, kind) // 2))


def _wgrad_ws(s):
    return _empty(tc.wgrad_bf16_workspace_size(s) // 4 + 4, dtype=F32)


# ------------------------------------------------------------------- prepare
def prepare(case, seed):
    kind, i = case["kind"], _inputs(case, seed)
    st = dict(kind=kind, i=i)
    if kind == "block":
        ss = st["s"] = _block_shapes(case)
        st["wf"] = [_packed(s, tc.OPERAND_FWD) for s in ss]
        st["wd"] = [_packed(s, tc.OPERAND_DGRAD) for s in ss]
        st["prep"] = tc.Prep([dict(layout=cg.NHWC, shape=s, weights=w, packed_fwd=f, packed_dgrad=d)
                              for s, w, f, d in zip(ss, i["w"], st["wf"], st["wd"])])
        st["a"] = [_empty(s.b, s.ho, s.wo, s.kn) for s in ss]
        st["dx"] = [_empty(s.b, s.h, s.w, s.c) for s in ss]
        st["dw"] = [torch.empty_like(w) for w in i["w"]]
        st["db"] = [_empty(s.kn, dtype=F32) for s in ss[:2]]
        st["ws"] = [_wgrad_ws(s) for s in ss]
        st["wsd"] = [_empty(cg.lib().convgemm_dgrad_bf16_bias_grad_workspace_size(s) // 4 + 4, dtype=F32) for s in ss]
        return st
    if kind == "group":
        convs = []
        for d, t in zip(_group_convs(case), i):
            s = _group_shape(d)
            wp = _empty(tc.group_weights_size(s) // 2)
            tc.group_pack_weights(cg.NHWC, s, t["w"], wp)
            convs.append(dict(shape=s, x=t["x"], w=wp, y=_empty(s.b, s.ho, s.wo, s.kn), shift=t["bias"], relu=True))
        st["group"], st["y"] = tc.Group(convs), [c["y"] for c in convs]
        return st
    s = st["s"] = _shape(case)
    st["dims"] = (s.b, s.h, s.w, s.c)
    if kind == "f32_host":
        st["y"] = np.empty((s.b, s.ho, s.wo, s.kn), np.float32)
        return st
    yshape = (s.b, s.ho, s.wo, s.kn)
    if kind == "f32":
        st["layout"] = cg.NCHW if case["layout"] == "nchw" else cg.NHWC
        st.update(y=torch.empty_like(i["dy"]), dx=torch.empty_like(i["x"]), dw=torch.empty_like(i["w"]),
                  ws=_empty(cg.wgrad_f32_workspace_size(s) // 4 + 4, dtype=F32))
        return st
    if kind == "torch":
        i["x"].requires_grad_()
        i["w"].requires_grad_()
        st["conf"] = (case["stride"], s.vpad, case["dil"], True)
        return st
    st["y"] = _empty(*yshape, dtype=F32 if kind == "bf16x3" else BF16)
    st["scale"], st["shift"] = _empty(s.kn, dtype=F32), _empty(s.kn, dtype=F32)
    if kind in ("infer", "fp8", "bf16x3"):
        tc.fold_epilogue(s.kn, st["scale"], st["shift"], i["bias"], i["mean"], i["inv_std"], i["gamma"], i["beta"])
    if kind == "infer":
        st["wp"] = _packed(s, tc.OPERAND_FWD)
        tc.pack_weights(cg.NHWC, s, tc.OPERAND_FWD, i["w"], st["wp"])
    elif kind == "fp8":
        st["wp"], st["wscale"] = _empty(tc.fp8_weights_size(s), dtype=torch.uint8), _empty(s.kn, dtype=F32)
        tc.fp8_pack_weights(cg.NHWC, s, i["w"], st["wp"], st["wscale"])
        st.update(xq=_empty(i["x"].numel(), dtype=torch.uint8), xscale=_empty(2, dtype=F32),
                  oscale=_empty(s.kn, dtype=F32), oshift=_empty(s.kn, dtype=F32))
    elif kind == "bf16x3":
        st["wp"] = [_packed(s, tc.OPERAND_FWD) for _ in range(2)]
        tc.bf16x3_pack_weights(cg.NHWC, s, i["w"], *st["wp"])
        st["xs"] = [_empty(*st["dims"]) for _ in range(2)]
    else:   # stem, nchw
        st["wp"] = _packed(s, tc.OPERAND_FWD)
        st["xb"] = _empty(s.b, s.h, s.w, tc.c8(s.c))
        st["dw"], st["ws"] = torch.empty_like(i["w"]), _wgrad_ws(s)
        if kind == "stem":
            st["stats"] = _empty(2, s.kn, dtype=torch.float64)
            st["wst"] = _empty(tc.fwd_bf16_stats_workspace_size(s) // 8 + 2, dtype=torch.float64)
            st["z"] = _empty(*yshape)
            st["mean"], st["var"] = _empty(s.kn, dtype=F32), _empty(s.kn, dtype=F32)
        else:
            st["wpd"] = _packed(s, tc.OPERAND_DGRAD)
            st["prep"] = tc.Prep([dict(layout=cg.NCHW, shape=s, weights=i["w"], packed_fwd=st["wp"], packed_dgrad=st["wpd"])])
            st["dyb"], st["dx"] = _empty(*yshape), _empty(*st["dims"])
            st["db"] = _empty(s.kn, dtype=F32)
            st["wsb"] = _empty(cg.lib().convgemm_bias_grad_bf16_workspace_size(s) // 4 + 4, dtype=F32)
    return st


# ----------------------------------------------------------------------- run
def run(st):
    return _RUN[st["kind"]](st, st["i"])


def _run_infer(st, i):
    tc.fwd_bf16(st["s"], i["x"], st["wp"], st["y"], st["scale"], st["shift"], relu=True)
    return st["y"]


def _run_block(st, i):
    s, a, dx = st["s"], st["a"], st["dx"]
    st["prep"].launch()
    for n, x in enumerate((i["x"], a[0], a[1])):
        tc.fwd_bf16(s[n], x, st["wf"][n], a[n], None, i["bias"][n], relu=True)
    tc.wgrad_bf16(cg.NHWC, s[2], i["dy"], a[1], st["dw"][2], st["ws"][2])
    tc.dgrad_bf16_bias_grad(s[2], i["dy"], st["wd"][2], dx[2], st["db"][1], a[1], st["wsd"][2])
    tc.wgrad_bf16(cg.NHWC, s[1], dx[2], a[0], st["dw"][1], st["ws"][1])
    tc.dgrad_bf16_bias_grad(s[1], dx[2], st["wd"][1], dx[1], st["db"][0], a[0], st["wsd"][1])
    tc.wgrad_bf16(cg.NHWC, s[0], dx[1], i["x"], st["dw"][0], st["ws"][0])
    tc.dgrad_bf16(s[0], dx[1], st["wd"][0], dx[0])
    return dict(y=a[2], dx=dx, dw=st["dw"], db=st["db"])


def _run_stem(st, i):
    s = st["s"]
    tc.to_bf16_nhwc(cg.NCHW, s.b, s.c, s.h, s.w, i["x"], st["xb"])
    tc.pack_weights(cg.NHWC, s, tc.OPERAND_FWD, i["w"], st["wp"])
    tc.fwd_bf16_stats(s, st["xb"], st["wp"], st["z"], st["stats"], workspace=st["wst"])
    npix = s.b * s.ho * s.wo
    tc.bn_stats_fold(s.kn, st["stats"], npix, st["scale"], st["shift"], i["gamma"], i["beta"], batch_mean=st["mean"],
                     batch_var=st["var"])
    tc.bn_apply_bf16(npix, s.kn, st["z"], st["scale"], st["shift"], st["y"], relu=True)
    tc.wgrad_bf16(cg.NHWC, s, i["dy"], st["xb"], st["dw"], st["ws"])
    return dict(y=st["y"], dw=st["dw"], mean=st["mean"], var=st["var"])


def _run_nchw(st, i):
    s = st["s"]
    tc.to_bf16_nhwc(cg.NCHW, s.b, s.c, s.h, s.w, i["x"], st["xb"])
    tc.to_bf16_nhwc(cg.NCHW, s.b, s.kn, s.ho, s.wo, i["dy"], st["dyb"])
    st["prep"].launch()
    tc.fwd_bf16(s, st["xb"], st["wp"], st["y"], None, i["bias"], relu=True)
    tc.dgrad_bf16(s, st["dyb"], st["wpd"], st["dx"])
    tc.wgrad_bf16(cg.NCHW, s, st["dyb"], st["xb"], st["dw"], st["ws"])
    tc.bias_grad_bf16(s, st["dyb"], st["db"], st["wsb"])
    return dict(y=st["y"], dx=st["dx"], dw=st["dw"], db=st["db"])


def _run_fp8(st, i):
    s = st["s"]
    tc.fp8_quantize(i["x"], st["xq"], st["xscale"])
    tc.fp8_epilogue_scales(s.kn, st["scale"], st["shift"], st["wscale"], st["xscale"], st["oscale"], st["oshift"])
    tc.fwd_fp8(s, st["xq"], st["wp"], st["y"], st["oscale"], st["oshift"], relu=True)
    return st["y"]


def _run_bf16x3(st, i):
    tc.split_bf16x2(i["x"], *st["xs"])
    tc.fwd_bf16x3(st["s"], *st["xs"], *st["wp"], st["y"], st["scale"], st["shift"], relu=True)
    return st["y"]


def _run_group(st, i):
    st["group"].launch()
    return st["y"]


def _run_torch(st, i):
    y = torch.ops.convgemm.conv2d_nhwc(i["x"], i["w"], None, i["bias"], *st["conf"])
    dx, dw = torch.autograd.grad(y, (i["x"], i["w"]), i["dy"])
    return dict(y=y.detach(), dx=dx, dw=dw)


def _run_f32_host(st, i):
    s = st["s"]
    cg.sconvGemmNHWC("N", s.b, s.h, s.w, s.c, s.kn, s.kh, s.kw, s.vpad, s.hpad, 1, 1, 1, 1, i["w"], i["x"], st["y"],
                     i["bias"], relu=True)
    return st["y"]


def _run_f32(st, i):
    s, lay = st["s"], st["layout"]
    cg.fwd_f32(lay, s, i["w"], i["x"], st["y"], bias=i["bias"], relu=True)
    cg.dgrad_f32(lay, s, i["w"], i["dy"], st["dx"], accumulate=False)
    cg.wgrad_f32(lay, s, i["dy"], i["x"], st["dw"], st["ws"])
    return dict(y=st["y"], dx=st["dx"], dw=st["dw"])


_RUN = dict(infer=_run_infer, block=_run_block, stem=_run_stem, nchw=_run_nchw, fp8=_run_fp8, bf16x3=_run_bf16x3,
            group=_run_group, torch=_run_torch, f32_host=_run_f32_host, f32=_run_f32)


# --------------------------------------------------------- the same in FP64
# NHWC tensors and [c][kh][kw][kn] weights, one GEMM per filter tap.
def _windows(s, t):
    p = torch.nn.functional.pad(t, (0, 0, s.hpad, s.hpad + s.hstride, s.vpad, s.vpad + s.vstride))
    for a in range(s.kh):
        for b in range(s.kw):
            y0, x0 = a * s.vdil, b * s.hdil
            yield a, b, p, (slice(None), slice(y0, y0 + (s.ho - 1) * s.vstride + 1, s.vstride),
                            slice(x0, x0 + (s.wo - 1) * s.hstride + 1, s.hstride))


def _fwd64(s, x, w, scale=None, shift=None, relu=True):
    y = torch.zeros(s.b * s.ho * s.wo, s.kn, dtype=torch.float64, device=x.device)
    for a, b, p, at in _windows(s, x):
        y.addmm_(p[at].reshape(-1, s.c), w[:, a, b, :])
    y = y if scale is None else y * scale
    y = y if shift is None else y + shift
    return (y.relu_() if relu else y).view(s.b, s.ho, s.wo, s.kn)


def _dgrad64(s, dy, w):
    g = dy.reshape(-1, s.kn)
    dx = torch.zeros(s.b, s.h, s.w, s.c, dtype=torch.float64, device=dy.device)
    for a, b, p, at in _windows(s, dx):
        if a == b == 0:
            acc = p
        acc[at] += (g @ w[:, a, b, :].t()).view(s.b, s.ho, s.wo, s.c)
    return acc[:, s.vpad:s.vpad + s.h, s.hpad:s.hpad + s.w].contiguous()


def _wgrad64(s, dy, x):
    dw = torch.zeros(s.c, s.kh, s.kw, s.kn, dtype=torch.float64, device=x.device)
    for a, b, p, at in _windows(s, x):
        dw[:, a, b, :] = p[at].reshape(-1, s.c).t() @ dy.reshape(-1, s.kn)
    return dw


def exact(case, seed):
    kind, i = case["kind"], _inputs(case, seed)
    if kind == "group":
        return [_fwd64(_group_shape(d), t["x"].double(), t["w"].double(), shift=t["bias"].double())
                for d, t in zip(_group_convs(case), i)]
    if kind == "f32_host":
        i = {k: torch.from_numpy(v).cuda() for k, v in i.items()}
    d = {k: [t.double() for t in v] if isinstance(v, list) else v.double() for k, v in i.items()}
    if kind == "block":
        s = _block_shapes(case)
        a = [d["x"]]
        for n in range(3):
            a.append(_fwd64(s[n], a[n], d["w"][n], shift=d["bias"][n]))
        g, dx, dw = d["dy"], [None] * 3, [None] * 3
        for n in (2, 1, 0):
            dw[n] = _wgrad64(s[n], g, a[n])
            g = dx[n] = _dgrad64(s[n], g, d["w"][n]) * (a[n] > 0 if n else 1)
        return dict(y=a[3], dx=dx, dw=dw, db=[dx[1].sum((0, 1, 2)), dx[2].sum((0, 1, 2))])
    s = _shape(case)
    nchw = kind == "nchw" or case.get("layout") == "nchw"
    x, w, dy = d["x"], d["w"], d.get("dy")
    if nchw or kind == "stem":
        x = x.permute(0, 2, 3, 1).contiguous()
    if nchw:
        w, dy = w.permute(1, 2, 3, 0).contiguous(), dy.permute(0, 2, 3, 1).contiguous()
    if kind in ("infer", "fp8", "bf16x3"):
        scale = d["gamma"] * d["inv_std"]
        return _fwd64(s, x, w, scale, d["beta"] + (d["bias"] - d["mean"]) * scale)
    if kind == "stem":
        z = _fwd64(s, x, w, relu=False)
        mean, var = z.mean((0, 1, 2)), z.var((0, 1, 2), unbiased=False)
        scale = d["gamma"] / (var + 1e-5).sqrt()
        return dict(y=((z - mean) * scale + d["beta"]).relu_(), dw=_wgrad64(s, dy, x), mean=mean, var=var)
    y = _fwd64(s, x, w, shift=d["bias"])
    if kind == "f32_host":
        return y
    g = dy * (y > 0) if kind == "torch" else dy
    out = dict(y=y, dx=_dgrad64(s, g, w), dw=_wgrad64(s, g, x))
    if kind == "nchw":   # BF16 tensors stay NHWC, the weight gradient comes in the NCHW API's layout
        out.update(dw=out["dw"].permute(3, 0, 1, 2).contiguous(), db=dy.sum((0, 1, 2)))
    elif nchw:
        out = dict(y=y.permute(0, 3, 1, 2).contiguous(), dx=out["dx"].permute(0, 3, 1, 2).contiguous(),
                   dw=out["dw"].permute(3, 0, 1, 2).contiguous())
    return out

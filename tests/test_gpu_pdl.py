"""GPU test of programmatic dependent launches: a chain of the library's small and large kernels, each reading what the
one before wrote into buffers that every round of the chain uses again, gives the same bits with the launches'
overlap on and off, enqueued eagerly without a pause and replayed from a captured graph."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

BF16 = torch.bfloat16


class Chain:
    """Conversion, packing, statistics, normalisation, gradients, quantisation and the precision forms of one layer."""

    def __init__(self, cg, b, hw, c, kn, k, stride):
        from convgemm_gb300 import tc
        self.cg, self.tc = cg, tc
        s = self.s = cg.Shape.of(b, hw, hw, c, kn, k, k, k // 2, k // 2, stride, stride)
        new = lambda *shape, dtype=BF16: torch.zeros(*shape, dtype=dtype, device="cuda")  # noqa: E731
        f32 = torch.float32
        self.x32, self.w32, self.dy32 = new(b, c, hw, hw, dtype=f32), new(kn, c, k, k, dtype=f32), new(b, kn, s.ho, s.wo, dtype=f32)
        self.x, self.dy, self.y, self.z, self.dx = new(b, hw, hw, c), new(b, s.ho, s.wo, kn), new(b, s.ho, s.wo, kn), new(b, s.ho, s.wo, kn), new(b, hw, hw, c)
        self.wf, self.wd = (new(tc.weights_size(s, op) // 2) for op in (tc.OPERAND_FWD, tc.OPERAND_DGRAD))
        self.pf, self.pd = torch.zeros_like(self.wf), torch.zeros_like(self.wd)
        self.sc, self.sh, self.mean, self.db, self.dbx = new(kn, dtype=f32), new(kn, dtype=f32), new(kn, dtype=f32), new(kn, dtype=f32), new(c, dtype=f32)
        self.stats, self.dz = new(2, kn, dtype=torch.float64), new(b, s.ho, s.wo, kn)
        self.dw, self.ws = new(kn * c * k * k, dtype=f32), new(tc.wgrad_bf16_workspace_size(s) // 4 + 4, dtype=f32)
        n1 = tc.fwd_bf16_stats_workspace_size(s)
        import ctypes
        n2 = cg.lib().convgemm_dgrad_bf16_bias_grad_workspace_size(ctypes.byref(s))
        n3 = cg.lib().convgemm_bias_grad_bf16_workspace_size(ctypes.byref(s))
        self.ws1, self.ws2, self.ws3 = new(n1 // 8 + 2, dtype=torch.float64), new(n2 // 4 + 4, dtype=f32), new(n3 // 4 + 4, dtype=f32)
        self.outs = [self.y, self.z, self.dx, self.dw, self.db, self.dbx, self.dz, self.stats, self.pf, self.pd]
        self.prep = tc.Prep([dict(layout=cg.NCHW, shape=s, weights=self.w32, packed_fwd=self.pf, packed_dgrad=self.pd)])
        self.grp_y = new(b, s.ho, s.wo, kn)
        self.gw = new(tc.group_weights_size(s) // 2)
        self.grp = tc.Group([dict(shape=s, x=self.x, w=self.gw, y=self.grp_y, scale=self.sc, shift=self.sh, relu=True)])
        self.outs.append(self.grp_y)
        if c % 64 == 0:
            self.q, self.qs = new(b, hw, hw, c, dtype=torch.uint8), new(2, dtype=f32)
            self.wq, self.wqs = new(tc.fp8_weights_size(s), dtype=torch.uint8), new(kn, dtype=f32)
            self.o1, self.o2, self.y8 = new(kn, dtype=f32), new(kn, dtype=f32), new(b, s.ho, s.wo, kn)
            self.xn = new(b, hw, hw, c, dtype=f32)
            self.hi, self.lo, self.wh, self.wl, self.y3 = new(b, hw, hw, c), new(b, hw, hw, c), torch.zeros_like(self.wf), torch.zeros_like(self.wf), new(b, s.ho, s.wo, kn, dtype=f32)
            self.outs += [self.q, self.y8, self.y3]

    def enqueue(self):
        cg, tc, s, N = self.cg, self.tc, self.s, self.cg.NCHW
        tc.to_bf16_nhwc(N, s.b, s.c, s.h, s.w, self.x32, self.x)
        tc.to_bf16_nhwc(N, s.b, s.kn, s.ho, s.wo, self.dy32, self.dy)
        tc.pack_weights(N, s, tc.OPERAND_FWD, self.w32, self.wf)
        tc.pack_weights(N, s, tc.OPERAND_DGRAD, self.w32, self.wd)
        self.prep.launch()
        tc.fwd_bf16_stats(s, self.x, self.pf, self.z, self.stats, workspace=self.ws1)
        tc.bn_stats_fold(s.kn, self.stats, s.b * s.ho * s.wo, self.sc, self.sh, batch_mean=self.mean)
        tc.bn_apply_bf16(s.b * s.ho * s.wo, s.kn, self.z, self.sc, self.sh, self.z)
        tc.fwd_bf16(s, self.x, self.wf, self.y, self.sc, self.sh, relu=True)
        tc.epilogue_grad_bf16(s.b * s.ho * s.wo, s.kn, self.dy, self.y, self.sc, self.dz)
        tc.bias_grad_bf16(s, self.dz, self.db, self.ws3)
        tc.dgrad_bf16_bias_grad(s, self.dz, self.pd, self.dx, self.dbx, relu_x=self.x, workspace=self.ws2)
        tc.dgrad_bf16_ex(s, self.dy, self.wd, self.dx, accumulate=True)
        tc.wgrad_bf16(N, s, self.dz, self.x, self.dw, self.ws)
        tc.group_pack_weights(N, s, self.w32, self.gw)
        self.grp.launch()
        if s.c % 64 == 0:
            tc.fp8_quantize(self.x, self.q, self.qs)
            tc.fp8_pack_weights(N, s, self.w32, self.wq, self.wqs)
            tc.fp8_epilogue_scales(s.kn, self.sc, self.sh, self.wqs, self.qs, self.o1, self.o2)
            tc.fwd_fp8(s, self.q, self.wq, self.y8, self.o1, self.o2)
            self.xn.copy_(self.x32.permute(0, 2, 3, 1))
            tc.split_bf16x2(self.xn, self.hi, self.lo)
            tc.bf16x3_pack_weights(N, s, self.w32, self.wh, self.wl)
            tc.fwd_bf16x3(s, self.hi, self.lo, self.wh, self.wl, self.y3)


@pytest.mark.parametrize("b,hw,c,kn,k,stride", [(1, 14, 256, 256, 3, 1), (2, 9, 72, 136, 3, 2), (16, 56, 64, 64, 3, 1), (8, 60, 3 * 8, 96, 3, 1),
                                                (4, 56, 64, 256, 1, 1)])
def test_chain_keeps_its_bits(cglib, b, hw, c, kn, k, stride):
    chain = Chain(cglib, b, hw, c, kn, k, stride)
    g = torch.Generator(device="cuda").manual_seed(c + kn)
    rand = lambda t: torch.randn(t.shape, device="cuda", generator=g)  # noqa: E731
    inputs = [[rand(chain.x32), rand(chain.w32) * 0.05, rand(chain.dy32)] for _ in range(3)]

    def load(i):
        for dst, src in zip((chain.x32, chain.w32, chain.dy32), inputs[i]):
            dst.copy_(src)

    def rounds(enqueue):
        kept = []
        for i in range(3):   # without a pause between them
            load(i)
            enqueue()
            kept.append([t.clone() for t in chain.outs])
        torch.cuda.synchronize()
        cglib.check_device()
        return kept

    chain.enqueue()
    torch.cuda.synchronize()
    try:
        cglib.set_pdl(0)
        want = rounds(chain.enqueue)
        for on in (0, 1):
            cglib.set_pdl(on)
            stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.graph(graph, stream=stream):
                chain.enqueue()
            for run in (chain.enqueue, graph.replay):
                for got, ref in zip(rounds(run), want):
                    for n, (a, r) in enumerate(zip(got, ref)):
                        assert torch.equal(a.reshape(-1).view(torch.uint8), r.reshape(-1).view(torch.uint8)), (on, run, n)
    finally:
        cglib.set_pdl(-1)

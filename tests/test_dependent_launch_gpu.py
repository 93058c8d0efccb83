"""Training steps out of the kernels that start before the one ahead of them has ended: every buffer is read by one kernel and written
over by a later one, and the parameters that the last kernel of a step writes are read by the first ones of the next."""
import pytest
import torch

from coccl_b200 import _lib
from coccl_b200.ops import gemm as G

pytestmark = pytest.mark.gpu


class _Steps:
    def __init__(self, device, M, H, F, V, rms):
        g = torch.Generator(device="cuda").manual_seed(M + H)
        self.M, self.H, self.F, self.V, self.rms = M, H, F, V, rms

        def bf(*shape, scale=1.0):
            return (torch.randn(*shape, device=device, generator=g) * scale).to(torch.bfloat16)

        def zeros(*shape, dtype=torch.float32):
            return torch.zeros(*shape, dtype=dtype, device=device)
        sizes = [F * H, F, V * F, H, H]
        n = sum(sizes)
        self.n, self.start = n, bf(n, scale=0.05)
        self.param, self.master, self.m, self.v, self.grad = zeros(n, dtype=torch.bfloat16), zeros(n), zeros(n), zeros(n), zeros(n)
        w1, self.b1, w2, self.gamma, self.beta = self.param.split(sizes)
        self.w1, self.w2 = w1.view(F, H), w2.view(V, F)
        g1, self.gb1, g2, self.ggamma, self.gbeta = self.grad.split(sizes)
        self.g1, self.g2 = g1.view(F, H), g2.view(V, F)
        self.x = bf(M, H)
        self.ids, self.targets = (torch.randint(0, V, (M,), device=device, generator=g) for _ in range(2))
        b16 = torch.bfloat16
        self.y, self.z, self.h, self.logits = zeros(M, H, dtype=b16), zeros(M, F, dtype=b16), zeros(M, F, dtype=b16), zeros(M, V, dtype=b16)
        self.dh, self.dz, self.dy, self.dx = zeros(M, F, dtype=b16), zeros(M, F, dtype=b16), zeros(M, H, dtype=b16), zeros(M, H, dtype=b16)
        self.mean, self.rstd, self.sq, self.coef = zeros(M), zeros(M), zeros(1), zeros(1)
        self.table = zeros(V, H)
        lib = _lib.lib()
        self.norm_scratch = zeros(lib.cocclkLayerNormBwdGrid(M) * 2 * H)
        self.sum_scratch = zeros(lib.cocclkColSumBlocks(M) * F)
        self.sq_scratch = zeros(lib.cocclkSumSqBlocks(n))
        self.embed_scratch = zeros(lib.cocclkEmbedScratchBytes(M, H), dtype=torch.uint8)
        self.losses = zeros(4, M)

    def run(self, wait=lambda: None):
        lib, st = _lib.lib(), _lib.cur_stream
        M, H, F, V = self.M, self.H, self.F, self.V

        def call(name, *args):
            args = [a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args]
            _lib.check(getattr(lib, name)(*args, st()), name)
            wait()

        def product(a, b, out, **kw):
            G.gemm(a, b, out=out, **kw)
            wait()
        self.param.copy_(self.start)
        self.master.copy_(self.start)
        for t in (self.m, self.v, self.grad, self.table):
            t.zero_()
        wait()
        for step in range(1, 5):
            if self.rms:
                call("cocclkRmsNormFwd", self.x, None, self.gamma, self.y, None, self.rstd, M, H, 1e-5)
            else:
                call("cocclkLayerNormFwd", self.x, None, self.gamma, self.beta, self.y, None, self.mean, self.rstd, M, H, 1e-5)
            product(self.y, self.w1, self.z, bias=self.b1)
            call("cocclkGeluFwd", self.z, None, self.h, None, M * F, F)
            product(self.h, self.w2, self.logits)
            call("cocclkCrossEntropy", self.logits, self.targets, self.losses[step - 1], M, V, V, 1.0 / M)
            product(self.logits.t(), self.h.t(), self.g2)
            product(self.logits, self.w2.t(), self.dh)
            call("cocclkGeluBwd", self.dh, self.z, self.dz, M * F)
            call("cocclkColSum", self.dz, self.gb1, 0, self.sum_scratch, M, F)
            product(self.dz.t(), self.y.t(), self.g1)
            product(self.dz, self.w1.t(), self.dy)
            if self.rms:
                call("cocclkRmsNormBwd", self.dy, self.x, self.rstd, self.gamma, self.dz if H == F else None, self.dx, self.ggamma, 0,
                     self.norm_scratch, M, H)
            else:
                call("cocclkLayerNormBwd", self.dy, self.x, self.mean, self.rstd, self.gamma, None, self.dx, self.ggamma, self.gbeta, 0,
                     self.norm_scratch, M, H)
            call("cocclkEmbedBwd", self.dx, self.ids, self.embed_scratch, self.table, M, H, V)
            call("cocclkEmbedPositionsBwd", self.dx, self.table, 2, M // 2, H)
            call("cocclkSumSq", self.grad, 0, self.n, self.sq, 0, self.sq_scratch)
            call("cocclkClipCoef", self.sq, 1.0, 1.0, self.coef, None)
            call("cocclkAdam", self.master, self.m, self.v, self.grad, 0, self.param, self.n, 1e-2, 0.9, 0.95, 1e-8, 0.1, step, self.coef)
        return [t.clone() for t in (self.param, self.master, self.m, self.v, self.grad, self.table, self.losses, self.dx, self.logits)]


@pytest.mark.parametrize("M,H,F,V,rms", [(64, 64, 128, 128, False), (256, 512, 1024, 1024, False), (200, 320, 320, 776, True),
                                         (1024, 1024, 512, 2048, True), (96, 9216, 64, 128, False)])
def test_steps_of_dependent_kernels(cuda, M, H, F, V, rms):
    """Launched back to back, and replayed from a graph: bit for bit what they give with a wait behind every launch."""
    steps = _Steps(cuda, M, H, F, V, rms)
    want = steps.run(torch.cuda.synchronize)
    assert all(bool(torch.isfinite(t.float()).all()) for t in want)
    assert not torch.equal(want[0], steps.start)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(steps.run(), want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = steps.run()
    for _ in range(5):
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("T,norm", [(384, True), (384, False), (1408, True), (1408, False)])
def test_rows_of_llama_kernels(cuda, T, norm):
    """The gate and the rotation, forward and backward, in a chain through their own results, on both sides of the rule by which a
    rotation without norms starts early."""
    S, nh, nkv, d, F = 128, 4, 2, 64, 512
    W = (nh + 2 * nkv) * d
    g = torch.Generator(device="cuda").manual_seed(9)

    def bf(*shape):
        return torch.randn(*shape, device=cuda, generator=g).to(torch.bfloat16)
    angle = torch.rand(S, d, device=cuda, generator=g)   # a row serves the first d / 2 of its values
    cos, sin = torch.cos(angle), torch.sin(angle)
    start, gates, wq, wk = bf(T, W), bf(T, 2 * F), *((bf(d), bf(d)) if norm else (None, None))
    lib = _lib.lib()
    q, k, v, dqkv = (torch.empty(T, n * d, dtype=torch.bfloat16, device=cuda) for n in (nh, nkv, nkv, nh + 2 * nkv))
    y, z = torch.empty(T, F, dtype=torch.bfloat16, device=cuda), torch.empty(T, 2 * F, dtype=torch.bfloat16, device=cuda)
    dq, dk = torch.zeros(d, device=cuda), torch.zeros(d, device=cuda)
    scratch = torch.zeros(lib.cocclkRotateBwdGrid(T) * 2 * d, device=cuda)
    sums = (dq, dk, 1, scratch) if norm else (None, None, 0, None)

    def run(wait=lambda: None):
        def call(name, *args):
            args = [a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args]
            _lib.check(getattr(lib, name)(*args, _lib.cur_stream()), name)
            wait()
        dqkv.copy_(start)
        z.copy_(gates)
        dq.zero_()
        dk.zero_()
        wait()
        for _ in range(3):   # the gradients of one turn are the values of the next
            call("cocclkRotateFwd", dqkv, q, k, v, cos, sin, wq, wk, T, S, nh, nkv, d, 1e-6)
            call("cocclkRotateBwd", q, k, v, start, dqkv, cos, sin, wq, wk, *sums, T, S, nh, nkv, d, 1e-6)
            call("cocclkSwigluFwd", z, y, T, F)
            call("cocclkSwigluBwd", y, gates, z, T, F)
        return [t.clone() for t in (q, k, v, dqkv, y, z, dq, dk)]
    want = run(torch.cuda.synchronize)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(run(), want))

"""Small outputs: the GEMM that splits the contraction over a cluster."""
import pytest
import torch

from coccl_b200.ops import gemm as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (65, 64, 72), (128, 72, 512), (130, 264, 1024), (65, 256, 4160), (200, 1000, 4096),
                                   (512, 2048, 2048), (1000, 1032, 1016), (513, 1544, 520)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (True, True), (False, True)])
def test_small_outputs_all_epilogues(cuda, M, N, K, a_mn, b_mn):
    """Outputs that the cluster kernel takes (1, 2, 4 and 8 ranks, ranks without a part of the contraction, ragged tiles and
    contractions) against 64 bits: fp32 sums of K products, whatever the split; and bit for bit the same twice."""
    if a_mn:
        M = -(-M // 8) * 8
    assert G.get_variant() == "auto"
    torch.manual_seed(M + N + K)
    a = torch.randn(K, M, device=cuda).to(torch.bfloat16).t() if a_mn else torch.randn(M, K, device=cuda).to(torch.bfloat16)
    b = torch.randn(K, N, device=cuda).to(torch.bfloat16).t() if b_mn else torch.randn(N, K, device=cuda).to(torch.bfloat16)
    bias = torch.randn(N, device=cuda).to(torch.bfloat16)
    ref = a.double() @ b.double().t()
    # the tensor core adds 16 products at a time to the fp32 accumulator and cuts the result off (2^-22 of its size, which the
    # sum of the products' sizes bounds), then up to 8 partial sums are added
    tol = (K / 16 + 8) * 2.0 ** -22 * (a.double().abs() @ b.double().abs().t())
    y = G.gemm(a, b, out_dtype=torch.float32)
    assert ((y.double() - ref).abs() <= tol).all()
    assert torch.equal(y, G.gemm(a, b, out_dtype=torch.float32))
    acc = torch.ones(M, N, device=cuda)
    G.gemm(a, b, out=acc, accumulate=True)
    assert ((acc.double() - 1 - ref).abs() <= tol + 2.0 ** -23 * (ref.abs() + 1)).all()
    o = G.gemm(a, b)
    assert ((o.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + tol).all()
    act, z = G.gemm(a, b, bias=bias, gelu=True, save_preact=True)
    want = ref + bias.double()
    assert ((z.double() - want).abs() <= 2.0 ** -8 * want.abs() + tol).all()
    gelu = torch.nn.functional.gelu(want, approximate="tanh")
    assert ((act.double() - gelu).abs() <= 2.0 ** -8 * gelu.abs() + 2 * tol + 2e-3 * want.abs()).all()   # tanh.approx: 2^-10.987
    # a pitch that rules the vector stores out goes to the other kernels, and comes out the same
    wide = torch.zeros(M, N + 8, device=cuda)
    G.gemm(a, b, out=wide[:, :N])
    assert ((wide[:, :N].double() - ref).abs() <= tol).all() and (wide[:, N:] == 0).all()
    G.check_errors()


@pytest.mark.parametrize("M,N,K,grad", [(8, 16384, 1024, True), (8, 16384, 1024, False), (8, 8192, 1024, True), (136, 8192, 1024, True),
                                        (8, 8192, 2048, False), (1024, 64, 64, True), (512, 2048, 2048, True), (512, 512, 4096, False)])
def test_the_rule_picks_no_kernel_that_is_far_behind(cuda, M, N, K, grad):
    """The kernel chosen by size against the single-CTA one (few rows of a weight gradient took 2.5 times as long on the wrong
    one), also where the small tiles are far ahead."""
    if grad:
        a, b = (torch.randn(K, n, device=cuda).to(torch.bfloat16).t() for n in (M, N))
        out = torch.zeros(M, N, device=cuda)

        def call():
            G.gemm(a, b, out=out, accumulate=True)
    else:
        a, b = (torch.randn(n, K, device=cuda).to(torch.bfloat16) for n in (M, N))
        out = torch.zeros(M, N, device=cuda, dtype=torch.bfloat16)

        def call():
            G.gemm(a, b, out=out)

    def us(variant):
        G.set_variant(variant)
        try:
            call()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                for _ in range(20):
                    call()
        finally:
            G.set_variant("auto")
        best = float("inf")
        for _ in range(5):
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            s.record()
            g.replay()
            e.record()
            e.synchronize()
            best = min(best, s.elapsed_time(e) / 20 * 1e3)
        return best
    single, auto = us("1cta"), us("auto")
    assert auto <= 1.25 * single, (auto, single)
    G.check_errors()

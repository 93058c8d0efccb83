"""Trainer kernels against PyTorch fp32 references."""
import dataclasses

import pytest
import torch
import torch.nn.functional as F

from coccl_b200 import _lib
from coccl_b200.ops import fused

pytestmark = pytest.mark.gpu


def test_layernorm_fwd_bwd(cuda):
    torch.manual_seed(0)
    M, H = 300, 1024
    x = torch.randn(M, H, device=cuda, dtype=torch.bfloat16, requires_grad=True)
    r = torch.randn(M, H, device=cuda, dtype=torch.bfloat16, requires_grad=True)
    g = (1 + 0.1 * torch.randn(H, device=cuda)).to(torch.bfloat16).requires_grad_(True)
    b = (0.1 * torch.randn(H, device=cuda)).to(torch.bfloat16).requires_grad_(True)
    y, xs = fused.layer_norm(x, g, b, 1e-5, residual=r)
    dy = torch.randn_like(y)
    dxs = torch.randn_like(xs)
    (y.float() * dy.float()).sum().add((xs.float() * dxs.float()).sum()).backward()
    xr, rr, gr, br = (t.detach().float().requires_grad_(True) for t in (x, r, g, b))
    xsr = (xr + rr).detach().to(torch.bfloat16).float() + (xr + rr) - (xr + rr).detach()
    yr = F.layer_norm(xsr, (H,), gr, br, 1e-5)
    ((yr * dy.float()).sum() + (xsr * dxs.float()).sum()).backward()
    assert torch.allclose(y.float(), yr, atol=3e-2, rtol=2e-2)
    assert torch.allclose(x.grad.float(), xr.grad, atol=5e-2, rtol=3e-2)
    assert torch.allclose(r.grad.float(), rr.grad, atol=5e-2, rtol=3e-2)
    assert torch.allclose(g.grad.float(), gr.grad, atol=0.5, rtol=3e-2)
    assert torch.allclose(b.grad.float(), br.grad, atol=0.5, rtol=3e-2)


def test_linear_gelu_fwd_bwd_with_main_grad(cuda):
    torch.manual_seed(1)
    M, K, N = 512, 256, 768
    x = (torch.randn(M, K, device=cuda) * 0.5).to(torch.bfloat16).requires_grad_(True)
    w = (torch.randn(N, K, device=cuda) * 0.05).to(torch.bfloat16).requires_grad_(True)
    bias = (torch.randn(N, device=cuda) * 0.1).to(torch.bfloat16).requires_grad_(True)
    w.main_grad = torch.zeros(N, K, device=cuda)
    bias.main_grad = torch.zeros(N, device=cuda)
    y = fused.linear(x, w, bias, gelu=True)
    dy = torch.randn_like(y)
    y.backward(dy)
    xr, wr, br = (t.detach().float().requires_grad_(True) for t in (x, w, bias))
    yr = F.gelu(F.linear(xr, wr, br), approximate="tanh")
    yr.backward(dy.float())
    assert torch.allclose(y.float(), yr, atol=2e-2, rtol=2e-2)
    assert torch.allclose(x.grad.float(), xr.grad, atol=3e-2, rtol=3e-2)
    assert torch.allclose(w.main_grad, wr.grad, atol=0.3, rtol=3e-2)
    assert torch.allclose(bias.main_grad, br.grad, atol=0.3, rtol=3e-2)
    assert w.grad is None and bias.grad is None


def test_cross_entropy(cuda):
    torch.manual_seed(2)
    M, V = 257, 50304
    logits = (torch.randn(M, V, device=cuda) * 2).to(torch.bfloat16)
    tgt = torch.randint(0, V, (M,), device=cuda)
    tgt[5] = -1
    ref_in = logits.float().requires_grad_(True)
    ref = F.cross_entropy(ref_in, tgt, ignore_index=-1, reduction="sum") * 0.01
    ref.backward()
    lg = logits.clone().requires_grad_(True)
    loss = fused.cross_entropy(lg, tgt, 0.01)
    loss.backward()
    assert abs(loss.item() - ref.item()) < 2e-3 * abs(ref.item())
    assert torch.allclose(lg.grad.float(), ref_in.grad, atol=2e-4, rtol=2e-2)


def test_adam_and_norm(cuda):
    torch.manual_seed(3)
    n = 100003
    master = torch.randn(n, device=cuda)
    m = torch.zeros(n, device=cuda)
    v = torch.zeros(n, device=cuda)
    g = torch.randn(n, device=cuda)
    p = torch.empty(n, device=cuda, dtype=torch.bfloat16)
    ref = master.clone().requires_grad_(True)
    opt = torch.optim.AdamW([ref], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    ss = torch.zeros(1, device=cuda)
    coef = torch.ones(1, device=cuda)
    norm = torch.zeros(1, device=cuda)
    for step in range(1, 4):
        fused.sum_squares(g, ss)
        fused.clip_coef(ss, 1.0, 1.0, coef, norm)
        assert abs(norm.item() - g.norm().item()) < 1e-3 * g.norm().item()
        fused.adam_step(master, m, v, g, p, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=step,
                        grad_scale=coef)
        ref.grad = g * min(1.0, 1.0 / (g.norm().item() + 1e-6))
        opt.step()
    assert torch.allclose(master, ref.detach(), atol=1e-5, rtol=1e-4)
    assert torch.allclose(p.float(), master, atol=1e-2, rtol=1e-2)


def test_gpt_step_matches_cpu_reference(cuda):
    """Tiny GPT: loss and gradients of the CUDA kernels path vs the fp32 CPU restatement of the same model."""
    from coccl_b200.models.gpt import GPTConfig, GPTStage
    cfg = GPTConfig(n_layer=2, hidden=256, n_head=4, ffn=1024, seq_len=128, vocab=1024)
    gpu = GPTStage(cfg, cuda, seed=5)
    cpu = GPTStage(dataclasses.replace(cfg, dtype=torch.float32), torch.device("cpu"), seed=5)
    cpu.store.flat_param.copy_(gpu.store.flat_param.float().cpu())
    torch.manual_seed(0)
    tok = torch.randint(0, cfg.vocab, (2, cfg.seq_len + 1))
    scale = 1.0 / (2 * cfg.seq_len)
    lg = gpu(tok[:, :-1].to(cuda), tok[:, 1:].to(cuda), scale)
    lg.backward()
    gpu.post_backward_sync_autograd_grads()
    lc = cpu(tok[:, :-1], tok[:, 1:], scale)
    lc.backward()
    cpu.post_backward_sync_autograd_grads()
    assert abs(lg.item() - lc.item()) < 2e-2
    a, b = gpu.store.flat_grad.cpu(), cpu.store.flat_grad
    rel = (a - b).norm() / b.norm()
    assert rel < 5e-2, rel.item()


@pytest.mark.parametrize("tp,M,V", [(2, 300, 1024), (4, 64, 25152)])
def test_vocab_parallel_cross_entropy_kernels(cuda, tp, M, V):
    """Two-pass cross-entropy over a vocabulary split into `tp` shards (all shards on this GPU): the combined loss and
    the in-place gradients equal the fp32 reference over the whole vocabulary."""
    import ctypes as C
    from coccl_b200 import _lib
    torch.manual_seed(21)
    full = (torch.randn(M, tp * V, device=cuda) * 3).to(torch.bfloat16)
    tgt = torch.randint(0, tp * V, (M,), device=cuda)
    tgt[::7] = -1   # ignored rows
    scale = 0.37
    shards = [full[:, r * V:(r + 1) * V].contiguous() for r in range(tp)]
    lib = _lib.lib()
    stats = torch.empty(tp, M, 4, dtype=torch.float32, device=cuda)
    for r in range(tp):
        _lib.check(lib.cocclkCrossEntropyStats(shards[r].data_ptr(), tgt.data_ptr(), stats[r].data_ptr(), M, V, V, r * V,
                                               _lib.cur_stream()), "stats")
    losses = []
    for r in range(tp):
        loss = torch.empty(M, dtype=torch.float32, device=cuda)
        _lib.check(lib.cocclkCrossEntropyFinish(shards[r].data_ptr(), tgt.data_ptr(), stats.data_ptr(), tp, loss.data_ptr(), M, V, V,
                                                r * V, scale, _lib.cur_stream()), "finish")
        losses.append(loss)
    lf = full.float()
    valid = tgt >= 0
    ref_loss = torch.where(valid, torch.logsumexp(lf, -1) - lf.gather(1, tgt.clamp(min=0)[:, None])[:, 0], torch.zeros(M, device=cuda))
    p = torch.softmax(lf, -1)
    p[torch.arange(M, device=cuda), tgt.clamp(min=0)] -= 1.0
    ref_grad = p * valid[:, None] * scale
    for r in range(tp):
        assert torch.allclose(losses[r], ref_loss, atol=2e-3, rtol=2e-3)
        assert torch.equal(losses[r], losses[0])   # every rank computes the same loss
        got = shards[r].float()
        want = ref_grad[:, r * V:(r + 1) * V]
        assert (got - want).abs().max().item() <= 4e-3 * scale + 1e-6


@pytest.mark.parametrize("M,N", [(4096, 4096), (100, 264), (2048, 6144), (33, 8)])
def test_column_sum(cuda, M, N):
    """Bias-gradient column sum (two kernels, fixed summation order) against fp32 torch, overwrite and accumulate."""
    import ctypes as C
    from coccl_b200 import _lib
    torch.manual_seed(22)
    x = torch.randn(M, N, device=cuda).to(torch.bfloat16)
    lib = _lib.lib()
    sc = torch.empty(lib.cocclkColSumBlocks(M) * N, dtype=torch.float32, device=cuda)
    out = torch.full((N,), 5.0, device=cuda)
    _lib.check(lib.cocclkColSum(x.data_ptr(), out.data_ptr(), 0, sc.data_ptr(), M, N, _lib.cur_stream()), "colsum")
    ref = x.float().sum(0)
    assert torch.allclose(out, ref, atol=1e-3 * M ** 0.5, rtol=1e-5)
    first = out.clone()
    _lib.check(lib.cocclkColSum(x.data_ptr(), out.data_ptr(), 1, sc.data_ptr(), M, N, _lib.cur_stream()), "colsum")
    assert torch.allclose(out, 2 * first, atol=1e-5, rtol=1e-6)   # same partial sums in the same order, added once more


@pytest.mark.parametrize("M,H", [(1, 8), (3, 264), (300, 512), (5, 2056), (297, 4096), (2, 16384)])
@pytest.mark.parametrize("residual", [False, True])
def test_rms_norm_kernels(cuda, M, H, residual):
    """Rows narrower than a warp, not a multiple of the CTA, several vectors a thread and the widest; fewer and more rows than
    the backward has CTAs. bf16 results carry a relative rounding error of 2^-9; the weight gradient sums M fp32 products."""
    from coccl_b200.models.llama import rms_norm
    torch.manual_seed(M + H)
    x = torch.randn(M, H, device=cuda).to(torch.bfloat16).requires_grad_(True)
    r = torch.randn(M, H, device=cuda).to(torch.bfloat16).requires_grad_(True) if residual else None
    w = (1 + 0.1 * torch.randn(H, device=cuda)).to(torch.bfloat16).requires_grad_(True)
    w.main_grad = torch.full((H,), 0.5, device=cuda)
    dy, dxs = (torch.randn(M, H, device=cuda).to(torch.bfloat16) for _ in range(2))
    assert fused.rms_norm_fits(x, w, r)
    if residual:
        y, xs = rms_norm(x, w, 1e-5, r)
        torch.autograd.backward([y, xs], [dy, dxs])
    else:
        y = rms_norm(x, w, 1e-5)
        y.backward(dy)
    s = (x + r if residual else x).detach().double().requires_grad_(True)
    wd = w.detach().double().requires_grad_(True)
    yr = s * torch.rsqrt(s.square().mean(-1, keepdim=True) + 1e-5) * wd
    yr.backward(dy.double())
    ds = s.grad + (dxs.double() if residual else 0)
    assert ((y.double() - yr).abs() <= 2 ** -8 * yr.abs() + 1e-5).all()
    assert ((x.grad.double() - ds).abs() <= 2 ** -8 * ds.abs() + 1e-4).all()
    assert not residual or torch.equal(x.grad, r.grad)
    assert w.grad is None
    assert torch.allclose(w.main_grad.double() - 0.5, wd.grad, rtol=1e-4, atol=1e-5 * M ** 0.5 + 1e-5)


def test_rms_norm_general_path_still_takes_the_rest(cuda):
    """fp32 tensors and rows that are not whole 16-byte vectors run as PyTorch operations."""
    from coccl_b200.models.llama import rms_norm
    for dtype, H in ((torch.float32, 64), (torch.bfloat16, 12)):
        x, w = torch.randn(5, H, device=cuda).to(dtype), torch.ones(H, device=cuda).to(dtype)
        assert not fused.rms_norm_fits(x, w)
        y, xs = rms_norm(x, w, 1e-5, x)
        assert torch.equal(xs, x + x)
        assert torch.allclose(y.float(), F.rms_norm((x + x).float(), (H,), w.float(), 1e-5), atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("M,F_", [(1, 8), (3, 520), (40, 2056), (2000, 264)])
def test_swiglu_kernels(cuda, M, F_):
    """One vector, ragged column blocks, more rows than CTAs; gates far enough out to saturate the sigmoid both ways."""
    torch.manual_seed(M)
    z = (torch.randn(M, 2 * F_, device=cuda) * 8).to(torch.bfloat16)
    z[0, :4] = torch.tensor([-300.0, 300.0, -80.0, 0.0])
    z.requires_grad_(True)
    dy = torch.randn(M, F_, device=cuda).to(torch.bfloat16)
    y = fused.swiglu(z)
    y.backward(dy)
    zd = z.detach().double().requires_grad_(True)
    g, u = zd.chunk(2, -1)
    yr = F.silu(g) * u
    yr.backward(dy.double())
    # one rounding to bf16 (2^-9); a flushed tail of the sigmoid is below 1e-30
    assert ((y.double() - yr).abs() <= 2 ** -8 * yr.abs() + 1e-30).all()
    assert ((z.grad.double() - zd.grad).abs() <= 2 ** -8 * zd.grad.abs() + 1e-5).all()


@pytest.mark.parametrize("d,nh,nkv", [(32, 3, 1), (64, 5, 5), (128, 32, 8), (128, 1, 1), (256, 6, 2)])
@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("batch,seq", [(1, 1), (2, 37), (1, 1300)])
def test_rotate_qkv_kernels(cuda, d, nh, nkv, norm, batch, seq):
    """Every head width the kernel takes, head counts that leave lanes idle, more tokens than CTAs; against the layer's own
    PyTorch operations in 64 bits. The weight gradients sum tokens x heads products in fp32."""
    from coccl_b200.models import llama
    torch.manual_seed(d + nh + seq)
    T = batch * seq
    qkv = torch.randn(T, (nh + 2 * nkv) * d, device=cuda).to(torch.bfloat16).requires_grad_(True)
    qw, kw = ((1 + 0.1 * torch.randn(d, device=cuda)).to(torch.bfloat16).requires_grad_(True) for _ in range(2)) if norm else (None, None)
    cos, sin = llama._rope_tables(seq, d, 1.0e4, cuda)
    assert fused.rotate_qkv_fits(qkv, d, qw, kw)
    out = fused.rotate_qkv(qkv, cos, sin, nh, nkv, qw, kw, 1e-5)
    grads = [torch.randn_like(o) for o in out]
    torch.autograd.backward(out, grads)

    def rms(x, w):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5) * w

    def rot(x):   # [batch, seq, heads, d]
        turned = torch.cat([-x[..., d // 2:], x[..., :d // 2]], -1)
        return x * cos.double()[:, None] + turned * sin.double()[:, None]
    xd = qkv.detach().double().requires_grad_(True)
    q, k, v = (t.view(batch, seq, -1, d) for t in xd.split([nh * d, nkv * d, nkv * d], -1))
    wd = [w.detach().double().requires_grad_(True) for w in (qw, kw)] if norm else []
    if norm:
        q, k = rms(q, wd[0]), rms(k, wd[1])
    ref = [t.reshape(T, -1, d) for t in (rot(q), rot(k), v)]
    torch.autograd.backward(ref, [g.double() for g in grads])
    # a rounding to bf16 of the result (2^-9); cancelling pairs leave an absolute error of a few fp32 steps
    for o, r in zip(out, ref):
        assert ((o.double() - r).abs() <= 2 ** -8 * r.abs() + 1e-5).all()
    assert ((qkv.grad.double() - xd.grad).abs() <= 2 ** -8 * xd.grad.abs() + 1e-4).all()
    for w, r in zip((qw, kw), wd):
        assert ((w.grad.double() - r.grad).abs() <= 2 ** -8 * r.grad.abs() + 1e-4 * (T * nh) ** 0.5).all()


@pytest.mark.parametrize("batch,seq,H", [(1, 1, 8), (2, 37, 1032), (2, 1024, 256), (1, 16384, 64)])
@pytest.mark.parametrize("ids_kind", ["random", "same", "distinct"])
def test_embedding_gradient_kernels(cuda, batch, seq, H, ids_kind):
    """One token, a ragged second column block, the largest batch; every id once, few ids, one id. Sums of up to 16384 bf16
    rows in fp32: the error of a sum of n terms of size 1 is at most n 2^-24 of the sum of their sizes."""
    torch.manual_seed(batch + seq)
    T, vocab = batch * seq, 20000
    ids = {"random": torch.randint(0, 50, (batch, seq), device=cuda), "same": torch.full((batch, seq), vocab - 1, device=cuda),
           "distinct": torch.randperm(vocab, device=cuda)[:T].view(batch, seq)}[ids_kind]
    wte = torch.randn(vocab, H, device=cuda).to(torch.bfloat16).requires_grad_(True)
    wpe = torch.randn(seq + 3, H, device=cuda).to(torch.bfloat16).requires_grad_(True)
    dy = torch.randn(T, H, device=cuda).to(torch.bfloat16)
    grads = []
    for _ in range(2):
        wte.main_grad, wpe.main_grad = torch.ones(vocab, H, device=cuda), torch.ones(seq + 3, H, device=cuda)
        assert fused.embed_fits(ids, wte, wpe, 2)
        e = fused.embed(ids, wte, wpe, 2)
        e.backward(dy)
        grads.append((wte.main_grad, wpe.main_grad))
    assert wte.grad is None and wpe.grad is None
    assert torch.equal(e, (wte[ids] + wpe[2:2 + seq]).reshape(T, H))
    assert torch.equal(grads[0][0], grads[1][0]) and torch.equal(grads[0][1], grads[1][1])
    g = torch.ones(vocab, H, device=cuda, dtype=torch.float64).index_add_(0, ids.reshape(-1), dy.double())
    size = torch.ones(vocab, H, device=cuda, dtype=torch.float64).index_add_(0, ids.reshape(-1), dy.double().abs())
    assert ((grads[0][0].double() - g).abs() <= T * 2.0 ** -24 * size + 1e-6).all()
    p = torch.ones(seq + 3, H, device=cuda, dtype=torch.float64)
    p[2:2 + seq] += dy.double().view(batch, seq, H).sum(0)
    assert ((grads[0][1].double() - p).abs() <= 1e-5).all()


def test_embedding_gradient_under_saved_tensor_hooks(cuda):
    """Hooks that pack and unpack every saved tensor (offloading) hand plain tensors back, without a `main_grad`."""
    wte = torch.randn(16, 8, device=cuda).to(torch.bfloat16).requires_grad_(True)
    wte.main_grad = torch.zeros(16, 8, device=cuda)
    ids = torch.tensor([[3, 3, 5]], device=cuda)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.cuda()):
        e = fused.embed(ids, wte)
    e.backward(torch.ones_like(e))
    assert wte.main_grad[3].tolist() == [2.0] * 8 and wte.main_grad[5].tolist() == [1.0] * 8 and wte.main_grad.sum() == 24


def test_embedding_beyond_the_sort_limit_takes_the_general_path(cuda):
    wte = torch.zeros(10, 8, device=cuda, dtype=torch.bfloat16).requires_grad_(True)
    wte.main_grad = torch.zeros(10, 8, device=cuda)
    assert fused.embed_fits(torch.zeros(2, 8192, dtype=torch.int64, device=cuda), wte)
    assert not fused.embed_fits(torch.zeros(2, 8193, dtype=torch.int64, device=cuda), wte)
    assert not fused.embed_fits(torch.zeros(2, 8, dtype=torch.int32, device=cuda), wte)


@pytest.mark.parametrize("M,V", [(1, 8), (3, 8200), (149, 50304), (297, 57344), (500, 1032)])
def test_cross_entropy_prefetched_rows(cuda, M, V):
    """One vector, fewer and more rows than SMs (one and several rows a CTA), the widest row; targets at both ends of a row and
    ignored ones. The gradient is p - 1{target} in fp32 with one rounding to bf16 (2^-9 of it)."""
    torch.manual_seed(M)
    logits = (torch.randn(M, V + 8, device=cuda) * 3).to(torch.bfloat16)[:, :V]   # a pitch larger than the row
    tgt = torch.randint(0, V, (M,), device=cuda)
    tgt[0], tgt[-1] = 0, V - 1
    if M > 2:
        tgt[1] = -100
    x = logits.double()
    loss = fused.cross_entropy(logits, tgt, 0.5)
    valid = tgt >= 0
    nll = torch.logsumexp(x, -1) - x.gather(1, tgt.clamp(min=0)[:, None])[:, 0]
    assert abs(loss.item() - 0.5 * nll[valid].sum().item()) <= 1e-5 * max(1.0, nll.sum().item())
    want = torch.softmax(x, -1)
    want[torch.arange(M, device=cuda), tgt.clamp(min=0)] -= 1
    want = want * valid[:, None] * 0.5
    assert ((logits.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()


@pytest.mark.parametrize("M,H", [(1, 8200), (2, 12288), (300, 8200), (149, 16384)])
@pytest.mark.parametrize("residual", [False, True])
def test_wide_layer_norm_backward(cuda, M, H, residual):
    """Rows that a CTA holds in parts (three and four vectors a thread, the last ones ragged), fewer and more rows than CTAs.
    bf16 results carry 2^-9; the weight gradients sum M fp32 products."""
    torch.manual_seed(M + H)
    x, dy, r = (torch.randn(M, H, device=cuda).to(torch.bfloat16) for _ in range(3))
    x.requires_grad_(True)
    g = (1 + 0.1 * torch.randn(H, device=cuda)).to(torch.bfloat16).requires_grad_(True)
    b = torch.randn(H, device=cuda).to(torch.bfloat16).requires_grad_(True)
    g.main_grad, b.main_grad = torch.full((H,), 0.5, device=cuda), torch.zeros(H, device=cuda)
    if residual:
        y, xs = fused.layer_norm(x, g, b, 1e-5, r)
        torch.autograd.backward([y, xs], [dy, r])
    else:
        fused.layer_norm(x, g, b, 1e-5).backward(dy)
    s = (x + r if residual else x).detach().double().requires_grad_(True)
    gd, bd = (t.detach().double().requires_grad_(True) for t in (g, b))
    F.layer_norm(s, (H,), gd, bd, 1e-5).backward(dy.double())
    ds = s.grad + (r.double() if residual else 0)
    assert ((x.grad.double() - ds).abs() <= 2 ** -8 * ds.abs() + 1e-4).all()
    assert torch.allclose(g.main_grad.double() - 0.5, gd.grad, rtol=1e-4, atol=1e-5 * M ** 0.5 + 1e-5)
    assert torch.allclose(b.main_grad.double(), bd.grad, rtol=1e-4, atol=1e-5 * M ** 0.5 + 1e-5)


def _device_us(fn, n=20):
    """Device time of one call of many, the least of five rounds."""
    for _ in range(3):
        fn()
    best = float("inf")
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(n):
            fn()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) / n * 1e3)
    return best


@pytest.mark.parametrize("rms", [False, True])
def test_norm_backward_has_no_cliff_at_wide_rows(cuda, rms):
    """One more vector a row must not cost several times the time (a kernel whose row does not fit the registers did: 20 times)."""
    lib, M = _lib.lib(), 4096

    def us(H):
        x, dy, dr = (torch.randn(M, H, device=cuda).to(torch.bfloat16) for _ in range(3))
        dx, g = torch.empty_like(x), torch.ones(H, device=cuda, dtype=torch.bfloat16)
        mean, rstd, dg, db = torch.zeros(M, device=cuda), torch.ones(M, device=cuda), torch.zeros(H, device=cuda), torch.zeros(H, device=cuda)
        sc = torch.empty(lib.cocclkLayerNormBwdGrid(M) * 2 * H, device=cuda)
        p = [t.data_ptr() for t in (dy, x, mean, rstd, g, dr, dx, dg, db, sc)]
        st = _lib.cur_stream()
        if rms:
            return _device_us(lambda: lib.cocclkRmsNormBwd(p[0], p[1], p[3], p[4], p[5], p[6], p[7], 1, p[9], M, H, st))
        return _device_us(lambda: lib.cocclkLayerNormBwd(*p[:9], 1, p[9], M, H, st))
    assert us(8200) <= 3 * us(8192)


@pytest.mark.parametrize("M,N", [(1, 16384), (129, 16384), (2049, 264), (4096, 2048), (64 * 32 + 1, 9472)])
def test_column_sum_block_rules(cuda, M, N):
    """Both folds (few and many partial rows, few and many columns) and both ends of the rule for the row blocks."""
    torch.manual_seed(M)
    x = torch.randn(M, N, device=cuda).to(torch.bfloat16)
    lib = _lib.lib()
    sc = torch.full((lib.cocclkColSumBlocks(M) * N + 8,), float("nan"), device=cuda)
    out = torch.ones(N, device=cuda)
    _lib.check(lib.cocclkColSum(x.data_ptr(), out.data_ptr(), 1, sc.data_ptr(), M, N, _lib.cur_stream()), "colsum")
    # fp32 sums of M terms of size 1
    assert ((out.double() - 1 - x.double().sum(0)).abs() <= M * 2.0 ** -24 * x.double().abs().sum(0) + 1e-6).all()
    assert sc[-8:].isnan().all()


def test_column_sum_of_wide_matrices_is_not_bound_by_its_fold(cuda):
    """A column sum of one row is two launches whatever its width (a fold with idle warps in a second wave took 1.5 times as long)."""
    lib = _lib.lib()

    def us(M, N):
        x, out = torch.zeros(M, N, device=cuda, dtype=torch.bfloat16), torch.zeros(N, device=cuda)
        sc = torch.empty(lib.cocclkColSumBlocks(M) * N, device=cuda)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(50):
                lib.cocclkColSum(x.data_ptr(), out.data_ptr(), 1, sc.data_ptr(), M, N, _lib.cur_stream())
        return _device_us(g.replay, 3) / 50
    assert us(1, 16384) <= 1.33 * us(1, 512)


@pytest.mark.parametrize("M,V", [(1, 8), (3, 2048), (593, 8192), (1300, 512), (600, 8200)])
def test_cross_entropy_narrow_rows(cuda, M, V):
    """The CTA of 256 threads: less than one vector a thread, the widest row it takes (and the first it does not), fewer and
    more rows than resident CTAs."""
    torch.manual_seed(M)
    logits = (torch.randn(M, V, device=cuda) * 3).to(torch.bfloat16)
    tgt = torch.randint(0, V, (M,), device=cuda)
    tgt[0], tgt[-1] = 0, V - 1
    if M > 2:
        tgt[1] = -1
    x = logits.double()
    loss = fused.cross_entropy(logits, tgt, 0.25)
    valid = tgt >= 0
    nll = torch.logsumexp(x, -1) - x.gather(1, tgt.clamp(min=0)[:, None])[:, 0]
    assert abs(loss.item() - 0.25 * nll[valid].sum().item()) <= 1e-5 * max(1.0, nll.sum().item())
    want = torch.softmax(x, -1)
    want[torch.arange(M, device=cuda), tgt.clamp(min=0)] -= 1
    want = want * valid[:, None] * 0.25
    assert ((logits.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()


def test_cross_entropy_of_narrow_rows_costs_less(cuda):
    """A sixteenth of the logits a row (with a whole SM for a row it took 0.84 of the time)."""
    lib = _lib.lib()

    def us(V):
        lg, tgt = torch.zeros(4096, V, device=cuda, dtype=torch.bfloat16), torch.zeros(4096, dtype=torch.int64, device=cuda)
        loss = torch.empty(4096, device=cuda)
        return _device_us(lambda: lib.cocclkCrossEntropy(lg.data_ptr(), tgt.data_ptr(), loss.data_ptr(), 4096, V, V, 1e-3, _lib.cur_stream()), 50)
    assert us(512) <= 0.66 * us(8192)


@pytest.mark.parametrize("H", [8, 1032])
@pytest.mark.parametrize("lengths", [(63, 64, 65), (1, 64, 64, 1, 128), (129, 130, 65, 65, 700), (7, 2000, 3)])
def test_embedding_gradient_of_long_runs(cuda, H, lengths):
    """Runs of equal ids around the length that is summed in one piece, long ones next to one another, their tokens shuffled."""
    torch.manual_seed(sum(lengths))
    T = sum(lengths)
    ids = torch.repeat_interleave(torch.arange(len(lengths), device=cuda) * 2, torch.tensor(lengths, device=cuda))
    ids = ids[torch.randperm(T, device=cuda)].view(1, T)
    wte = torch.zeros(2 * len(lengths), H, device=cuda, dtype=torch.bfloat16).requires_grad_(True)
    dy = torch.randn(T, H, device=cuda).to(torch.bfloat16)
    grads = []
    for _ in range(3):
        wte.main_grad = torch.ones(2 * len(lengths), H, device=cuda)
        fused.embed(ids, wte).backward(dy)
        grads.append(wte.main_grad)
    assert torch.equal(grads[0], grads[1]) and torch.equal(grads[0], grads[2])
    want = torch.ones(2 * len(lengths), H, device=cuda, dtype=torch.float64).index_add_(0, ids[0], dy.double())
    size = torch.ones_like(want).index_add_(0, ids[0], dy.double().abs())
    assert ((grads[0].double() - want).abs() <= T * 2.0 ** -24 * size + 1e-6).all()


@pytest.mark.parametrize("V,H", [(512, 128), (8192, 512)])
def test_embedding_gradient_of_padded_batches_costs_no_more(cuda, V, H):
    """Half of the tokens one id (padding) against all of them random (one CTA for a run took 6.5 times as long)."""
    wte = torch.zeros(V, H, device=cuda, dtype=torch.bfloat16).requires_grad_(True)
    wte.main_grad = torch.zeros(V, H, device=cuda)
    dy = torch.randn(16384, H, device=cuda).to(torch.bfloat16)
    us = []
    for padded in (False, True):
        ids = torch.randint(0, V, (2, 8192), device=cuda)
        if padded:
            ids[:, 4096:] = 0
        e = fused.embed(ids, wte)
        us.append(_device_us(lambda: e.backward(dy, retain_graph=True)))
    assert us[1] <= 2 * us[0], us

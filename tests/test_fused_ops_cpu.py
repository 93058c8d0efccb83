"""Host side of the fused training operations, with the kernel library replaced by a stand-in that reads what the kernels would
read (the pointers and sizes of each launch)."""
import ctypes
import math

import pytest
import torch
import torch.nn.functional as F

from coccl_b200 import _lib
from coccl_b200.models import llama
from coccl_b200.ops import fused


def _read(ptr, n, ctype, dtype):
    return torch.tensor((ctype * n).from_address(ptr)[:], dtype=dtype)


class EmbedKernels:
    """The embedding gradient as embed_kernels.cu computes it: `T` consecutive 64-bit ids, rows of dy back to back."""

    def __init__(self, tables):
        self.grads = {t.main_grad.data_ptr(): t.main_grad for t in tables}
        self.calls = []

    def cocclkEmbedScratchBytes(self, T, H):
        return 16 * T

    def cocclkEmbedBwd(self, dy, ids, scratch, grad, T, H, vocab, stream):
        self.calls.append("rows")
        rows = _read(dy, T * H, ctypes.c_uint16, torch.int32).to(torch.int16).view(torch.bfloat16).view(T, H)
        self.grads[grad].index_add_(0, _read(ids, T, ctypes.c_int64, torch.int64), rows.float())
        return 0

    def cocclkEmbedPositionsBwd(self, dy, grad, batch, seq, H, stream):
        self.calls.append("positions")
        rows = _read(dy, batch * seq * H, ctypes.c_uint16, torch.int32).to(torch.int16).view(torch.bfloat16).view(batch, seq, H)
        out = (ctypes.c_float * (seq * H)).from_address(grad)
        for i, v in enumerate(rows.float().sum(0).reshape(-1).tolist()):
            out[i] += v
        return 0


def _table(rows, H, seed):
    t = torch.nn.Parameter(torch.randn(rows, H, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16))
    t.main_grad = torch.zeros(rows, H)
    return t


@pytest.fixture
def embed_kernels(monkeypatch):
    wte, wpe = _table(40, 8, 1), _table(12, 8, 2)
    k = EmbedKernels([wte])
    monkeypatch.setattr(_lib, "lib", lambda: k)
    monkeypatch.setattr(_lib, "cur_stream", lambda: 0)
    return k, wte, wpe


@pytest.mark.parametrize("kind", ["plain", "column", "every other column", "transposed", "expanded"])
def test_embedding_gradient_follows_the_ids_whatever_their_strides(embed_kernels, kind):
    _, wte, wpe = embed_kernels
    tok = torch.randint(0, 40, (4, 10), generator=torch.Generator().manual_seed(3))
    ids = {"plain": tok, "column": tok[:, 2:3], "every other column": tok[:1, ::2], "transposed": tok.t(),
           "expanded": tok[:, :1].expand(4, 5)}[kind]
    e = fused.embed(ids, wte, wpe)
    assert torch.equal(e, (wte[ids] + wpe[:ids.shape[1]]).reshape(-1, 8))
    dy = torch.randn(e.shape, generator=torch.Generator().manual_seed(4)).to(torch.bfloat16)
    e.backward(dy)
    want = torch.zeros(40, 8).index_add_(0, ids.reshape(-1), dy.float())
    assert torch.allclose(wte.main_grad, want, atol=1e-5)


def _embedded(embed_kernels):
    """A pass through the tables with its gradients as autograd's own operations give them."""
    k, wte, wpe = embed_kernels
    ids = torch.tensor([[3, 3, 5], [0, 39, 5]])
    dy = torch.randn(6, 8, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16)
    a, b = (t.detach().clone().requires_grad_(True) for t in (wte, wpe))
    (F.embedding(ids, a) + b[2:5]).reshape(6, 8).backward(dy)
    return k, wte, wpe, fused.embed(ids, wte, wpe, 2), dy, a.grad, b.grad


def test_hooks_on_the_embedding_tables_see_and_change_the_gradient(embed_kernels):
    k, wte, wpe, e, dy, gw, gp = _embedded(embed_kernels)
    seen = []
    handles = [wte.register_hook(lambda g: (seen.append(g.clone()), g * 0)[1]), wpe.register_post_accumulate_grad_hook(seen.append)]
    e.backward(dy, retain_graph=True)
    assert not k.calls and torch.equal(seen[0], gw) and seen[1] is wpe
    assert torch.equal(wte.grad, torch.zeros_like(wte)) and torch.equal(wpe.grad, gp)
    for h in handles:
        h.remove()
    wte.grad = wpe.grad = None
    e.backward(dy)
    assert k.calls == ["rows", "positions"] and wte.grad is None and wpe.grad is None
    assert torch.allclose(wte.main_grad, gw.float(), atol=2e-2, rtol=1e-2) and torch.allclose(wpe.main_grad, gp.float(), atol=2e-2, rtol=1e-2)


def test_gradients_of_the_embedding_tables_can_be_asked_for(embed_kernels):
    k, wte, wpe, e, dy, gw, gp = _embedded(embed_kernels)
    a, b = torch.autograd.grad(e, (wte, wpe), dy, retain_graph=True)
    assert torch.equal(a, gw) and torch.equal(b, gp) and not k.calls
    e.backward(dy, inputs=[wpe], retain_graph=True)
    assert k.calls == ["positions"] and wte.grad is None
    # second derivatives: d/d(dy) of sum(gradient * c) is c looked up by the ids
    d2 = dy.clone().requires_grad_(True)
    (g,) = torch.autograd.grad(e, wte, d2, create_graph=True)
    c = torch.randn(40, 8, generator=torch.Generator().manual_seed(6)).to(torch.bfloat16)
    (back,) = torch.autograd.grad(g, d2, c)
    assert torch.equal(back, c[torch.tensor([3, 3, 5, 0, 39, 5])])


class LlamaKernels:
    """What the Llama kernels compute; the backward kernels of the rotation and the gate write nothing."""

    @staticmethod
    def _bf16(ptr, *shape):
        n = math.prod(shape)
        return torch.frombuffer((ctypes.c_uint8 * (2 * n)).from_address(ptr), dtype=torch.bfloat16).view(*shape)

    @staticmethod
    def _fp32(ptr, *shape):
        n = math.prod(shape)
        return torch.frombuffer((ctypes.c_uint8 * (4 * n)).from_address(ptr), dtype=torch.float32).view(*shape)

    def cocclkLayerNormBwdGrid(self, M):
        return 1

    cocclkRotateBwdGrid = cocclkLayerNormBwdGrid

    def __getattr__(self, name):
        if name.endswith("Bwd"):
            return lambda *a: 0
        raise AttributeError(name)

    def cocclkRmsNormFwd(self, x, res, w, y, xo, rstd, M, H, eps, stream):
        xs = self._bf16(x, M, H)
        if res:
            xs = self._bf16(xo, M, H).copy_(xs + self._bf16(res, M, H))
        r = torch.rsqrt(xs.float().square().mean(-1, keepdim=True) + eps)
        self._fp32(rstd, M, 1).copy_(r)
        self._bf16(y, M, H).copy_(xs.float() * r * self._bf16(w, H).float())
        return 0

    def cocclkRmsNormBwd(self, dy, x, rstd, w, dres, dx, dw, accumulate, scratch, M, H, stream):
        got = llama.rms_norm_gradients(self._bf16(x, M, H), self._bf16(w, H), self._fp32(rstd, M, 1), self._bf16(dy, M, H))
        self._bf16(dx, M, H).copy_(got[0] + (self._bf16(dres, M, H) if dres else 0))
        self._fp32(dw, H).copy_(got[1] + (self._fp32(dw, H) if accumulate else 0))
        return 0

    def cocclkRotateFwd(self, qkv, q, k, v, cos, sin, qw, kw, T, seq, nh, nkv, d, eps, stream):
        heads = self._bf16(qkv, T, nh + 2 * nkv, d).float()
        at = torch.arange(T) % seq
        c, s = (self._fp32(p, seq, d)[at][:, None] for p in (cos, sin))
        for out, x, w in ((q, heads[:, :nh], qw), (k, heads[:, nh:nh + nkv], kw)):
            if w:
                x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * self._bf16(w, d).float()
            self._bf16(out, *x.shape).copy_(x * c + torch.cat([-x[..., d // 2:], x[..., :d // 2]], -1) * s)
        self._bf16(v, T, nkv, d).copy_(heads[:, nh + nkv:])
        return 0

    def cocclkSwigluFwd(self, z, y, M, F_, stream):
        gate, up = self._bf16(z, M, 2 * F_).chunk(2, -1)
        self._bf16(y, M, F_).copy_(F.silu(gate.float()) * up.float())
        return 0


def _second(outputs, inputs, seed):
    """Gradients of `inputs` under create_graph and, from a random weighting of those, the gradients once more."""
    gen = torch.Generator().manual_seed(seed)
    dys = [torch.randn(o.shape, generator=gen).to(o.dtype).requires_grad_(True) for o in outputs]
    first = torch.autograd.grad(outputs, inputs, dys, create_graph=True)
    total = sum((g * torch.randn(g.shape, generator=gen).to(g.dtype)).sum() for g in first)
    second = torch.autograd.grad(total, [*inputs, *dys], allow_unused=True)
    return [*first, *(torch.zeros(()) if g is None else g for g in second)]


@pytest.mark.parametrize("case", ["norm", "norm + residual", "norm, rows apart", "rotation", "rotation + head norm", "gate"])
def test_gradients_of_the_llama_functions_can_be_differentiated(monkeypatch, case):
    """First and second derivatives against the same functions in 64 bits. bf16 results in a chain of a few operations: 2^-8 of
    the largest value in each."""
    k = LlamaKernels()
    monkeypatch.setattr(_lib, "lib", lambda: k)
    monkeypatch.setattr(_lib, "cur_stream", lambda: 0)
    gen = torch.Generator().manual_seed(11)

    def leaf(*shape):
        return torch.randn(*shape, generator=gen).to(torch.bfloat16).requires_grad_(True)
    eps, T, seq, nh, nkv, d = 1e-5, 6, 3, 2, 1, 8

    def rms(x, w):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w
    if case.startswith("norm"):
        x, w, r = leaf(5, 32), leaf(16), leaf(5, 16)
        inputs = [x, w] + ([r] if "residual" in case else [])
        xin = x[:, ::2] if "apart" in case else x[:, :16].contiguous()
        out = fused.rms_norm(xin, w, eps, r if "residual" in case else None)
        out = out if isinstance(out, tuple) else (out,)
        wide = [t.detach().double().requires_grad_(True) for t in inputs]
        xw = wide[0][:, ::2] if "apart" in case else wide[0][:, :16]
        xs = xw + wide[2] if "residual" in case else xw
        ref = (rms(xs, wide[1]), xs)[:len(out)]
    elif case.startswith("rotation"):
        x, qw, kw = leaf(T, (nh + 2 * nkv) * d), leaf(d), leaf(d)
        inputs = [x] + ([qw, kw] if "norm" in case else [])
        cos, sin = llama._rope_tables(seq, d, 100.0, torch.device("cpu"))
        out = fused.rotate_qkv(x, cos, sin, nh, nkv, *(inputs[1:] or (None, None)), eps)
        wide = [t.detach().double().requires_grad_(True) for t in inputs]
        heads = wide[0].view(T, -1, d)
        at = torch.arange(T) % seq
        parts = [heads[:, :nh], heads[:, nh:nh + nkv]]
        if "norm" in case:
            parts = [rms(p, w) for p, w in zip(parts, wide[1:])]
        ref = [p * cos.double()[at][:, None] + torch.cat([-p[..., d // 2:], p[..., :d // 2]], -1) * sin.double()[at][:, None]
               for p in parts] + [heads[:, nh + nkv:]]
    else:
        inputs = [leaf(4, 32)]
        out = (fused._Swiglu.apply(inputs[0]),)
        wide = [inputs[0].detach().double().requires_grad_(True)]
        gate, up = wide[0].chunk(2, -1)
        ref = (F.silu(gate) * up,)
    for got, want in zip(_second(out, inputs, 21), _second(ref, wide, 21)):
        assert (got.double() - want).abs().max() <= 3 * 2.0 ** -8 * max(1.0, want.abs().max().item())


@pytest.fixture
def llama_as_on_the_gpu(monkeypatch):
    """CPU tensors that the rules for the kernels take for CUDA ones; a kernel call fails."""
    class No:
        def __getattr__(self, name):
            raise AssertionError(f"{name} called")
    monkeypatch.setattr(_lib, "lib", lambda: No())
    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda t: True))


def _llama_functions():
    """(function of one bf16 tensor [4, 32], the same as PyTorch operations): what the Llama layers run on one tensor."""
    w, table = torch.linspace(0.5, 1.5, 32).to(torch.bfloat16), _table(40, 8, 1)
    return {"gate": (fused.swiglu, lambda z: F.silu(z[..., :16]) * z[..., 16:]),
            "embedding": (lambda x: fused.embed_fits((x.reshape(-1, 32)[:, :2] * 0).long(), table), None),
            "norm": (lambda x: fused.rms_norm_fits(x, w), None), "rotation": (lambda x: fused.rotate_qkv_fits(x, 32), None)}


@pytest.mark.parametrize("around", ["vmap", "forward mode", "dispatch mode", "subclass"])
@pytest.mark.parametrize("name", ["gate", "norm", "rotation", "embedding"])
def test_transforms_and_modes_work_on_operations(llama_as_on_the_gpu, around, name):
    from torch.utils._python_dispatch import TorchDispatchMode

    class Count(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Sub(torch.Tensor):
        pass
    fn, ref = _llama_functions()[name]
    x = torch.randn(4, 32, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16)
    if ref is None:   # a rule: yes for plain tensors, no here
        assert fn(x)
        if around == "vmap":
            assert torch.vmap(lambda t: t * (1 + int(fn(x))))(x).equal(x)
        elif around == "forward mode":
            with torch.autograd.forward_ad.dual_level():
                assert not fn(x)
        elif around == "dispatch mode":
            with Count():
                assert not fn(x)
        else:
            assert not fn(x.as_subclass(Sub))
        return
    if around == "vmap":
        assert torch.equal(torch.vmap(fn)(x), ref(x))
    elif around == "forward mode":
        got, want = (torch.func.jvp(f, (x,), (torch.ones_like(x),)) for f in (fn, ref))
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    elif around == "dispatch mode":
        with Count():
            assert torch.equal(fn(x), ref(x))
    else:
        assert torch.equal(fn(x.as_subclass(Sub)), ref(x))


@pytest.mark.parametrize("kind", ["one column", "every other column", "whole rows"])
def test_cross_entropy_reads_its_targets_whatever_their_strides(monkeypatch, kind):
    seen = []

    class K:
        def cocclkCrossEntropy(self, logits, targets, loss, M, V, ld, scale, stream):
            seen.append(_read(targets, M, ctypes.c_int64, torch.int64))
            return 0
    tok = torch.arange(40).view(4, 10)
    targets = {"one column": tok[:, 1:2], "every other column": tok[:1, ::2], "whole rows": tok}[kind]
    logits = torch.zeros(targets.numel(), 64, dtype=torch.bfloat16)
    monkeypatch.setattr(_lib, "lib", lambda: K())
    monkeypatch.setattr(_lib, "cur_stream", lambda: 0)
    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda t: True))
    fused.cross_entropy(logits, targets, 1.0)
    assert torch.equal(seen[0], targets.reshape(-1))

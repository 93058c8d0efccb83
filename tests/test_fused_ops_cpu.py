"""Host side of the fused training operations, with the kernel library replaced by a stand-in that reads what the kernels would
read (the pointers and sizes of each launch)."""
import ctypes

import pytest
import torch
import torch.nn.functional as F

from coccl_b200 import _lib
from coccl_b200.ops import fused


def _read(ptr, n, ctype, dtype):
    return torch.tensor((ctype * n).from_address(ptr)[:], dtype=dtype)


class EmbedKernels:
    """The embedding gradient as embed_kernels.cu computes it: `T` consecutive 64-bit ids, rows of dy back to back."""

    def __init__(self, tables):
        self.grads = {t.main_grad.data_ptr(): t.main_grad for t in tables}
        self.calls = []

    def cocclkEmbedOrder(self, ids, order, T, stream):
        self.calls.append("order")
        return 0

    def cocclkEmbedBwd(self, dy, ids, order, grad, T, H, vocab, stream):
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
    assert k.calls == ["order", "rows", "positions"] and wte.grad is None and wpe.grad is None
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

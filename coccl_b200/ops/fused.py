"""Autograd functions over the trainer kernels (csrc/kernels/train_kernels.cu,
gemm_kernels.cu). CUDA tensors always run the sm_100a kernels; CPU tensors run a
plain PyTorch restatement of the same math, which is what the multi-process
`gloo` tests of the parallel layers use (there is no GPU fallback path).

Weight gradients follow the Megatron convention: when a parameter carries a
`.main_grad` fp32 buffer, backward accumulates into it (wgrad GEMM with fp32
accumulate epilogue) and returns None for that parameter.
"""
from __future__ import annotations

import threading

import torch
import torch.nn.functional as F

from .. import _lib
from . import gemm as G

_scratch: dict[tuple, torch.Tensor] = {}


def scratch(device, nfloats: int, tag: str = "") -> torch.Tensor:
    """Per-device, per-tag fp32 scratch buffer that only ever grows (stream-ordered reuse)."""
    key = (device.index, tag)
    t = _scratch.get(key)
    if t is None or t.numel() < nfloats:
        t = torch.empty(max(nfloats, 1 << 16), dtype=torch.float32, device=device)
        _scratch[key] = t
    return t


class Branch:
    """A second stream for backward work that only ends in gradient buffers (weight and bias gradients, embedding tables) while a
    forward and backward pass is captured into a graph: small products fill a fraction of the GPU and nothing waits for these, yet
    in one stream they stand between the kernels that do wait for one another. All such work of a pass goes through one branch in
    its old order, so every buffer sees its sums in the order of the launched pass. The tensors it reads are kept until `join`:
    the allocator knows the main stream only and would hand their memory out again. Leaving the context joins, also on an error: a
    capture with a stream that has not come back cannot even be ended."""

    _of_thread = threading.local()

    def __init__(self, device):
        self.stream, self.keep, self.used = torch.cuda.Stream(device), [], False

    @classmethod
    def current(cls):
        """The branch of the pass that this thread is capturing (None: everything in one stream)."""
        return getattr(cls._of_thread, "branch", None)

    def __enter__(self):
        self._of_thread.branch = self
        return self

    def __exit__(self, error, *_):
        self._of_thread.branch = None
        try:
            self.join(torch.cuda.current_stream(self.stream.device))
        except RuntimeError:   # of a capture that the error in flight has broken
            if error is None:
                raise

    def run(self, work, *reads):
        """work() behind what the current stream holds so far, beside what it gets from now on."""
        self.stream.wait_stream(torch.cuda.current_stream(self.stream.device))
        self.keep.append(reads)
        self.used = True
        with torch.cuda.stream(self.stream):
            return work()

    def join(self, stream):
        try:
            if self.used:
                stream.wait_stream(self.stream)
        finally:
            self.keep = []


def _accum_param_grad(p: torch.Tensor, g_fp32_or_none, compute):
    """compute(out_fp32, accumulate) writes the gradient; returns what autograd should see."""
    mg = getattr(p, "main_grad", None)
    if mg is not None:
        compute(mg, True)
        return None
    out = torch.empty(p.shape, dtype=torch.float32, device=p.device)
    compute(out, False)
    return out.to(p.dtype)


# --------------------------------------------------------------------------- LayerNorm (+ residual add)
class _LayerNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, res, gamma, beta, eps):
        H = x.shape[-1]
        x2 = x.reshape(-1, H)
        M = x2.shape[0]
        has_res = res is not None
        if x.is_cuda:
            x2 = x2.contiguous()
            r2 = res.reshape(-1, H).contiguous() if has_res else None
            y = torch.empty_like(x2)
            xo = torch.empty_like(x2) if has_res else None
            mean = torch.empty(M, dtype=torch.float32, device=x.device)
            rstd = torch.empty(M, dtype=torch.float32, device=x.device)
            rc = _lib.lib().cocclkLayerNormFwd(x2.data_ptr(), _lib.ptr(r2), gamma.data_ptr(), beta.data_ptr(),
                                               y.data_ptr(), _lib.ptr(xo), mean.data_ptr(), rstd.data_ptr(), M, H,
                                               eps, _lib.cur_stream())
            _lib.check(rc, "cocclkLayerNormFwd")
            xs = xo if has_res else x2
        else:
            xs = (x2.float() + res.reshape(-1, H).float()).to(x.dtype) if has_res else x2
            xf = xs.float()
            mean = xf.mean(-1)
            rstd = torch.rsqrt(xf.var(-1, unbiased=False) + eps)
            y = (((xf - mean[:, None]) * rstd[:, None]) * gamma.float() + beta.float()).to(x.dtype)
        ctx.save_for_backward(xs, mean, rstd, gamma, beta)
        ctx.has_res = has_res
        ctx.shape = x.shape
        if has_res:
            return y.reshape(x.shape), xs.reshape(x.shape)
        return y.reshape(x.shape), None

    @staticmethod
    def backward(ctx, dy, dxs):
        xs, mean, rstd, gamma, beta = ctx.saved_tensors
        H = xs.shape[-1]
        M = xs.shape[0]
        dy2 = dy.reshape(-1, H)
        dres = dxs.reshape(-1, H) if dxs is not None else None
        if xs.is_cuda:
            dy2 = dy2.contiguous()
            dres = dres.contiguous() if dres is not None else None
            dx = torch.empty_like(xs)
            grid = _lib.lib().cocclkLayerNormBwdGrid(M)
            sc = scratch(xs.device, grid * 2 * H, "ln")

            def run(dg, db, acc):
                rc = _lib.lib().cocclkLayerNormBwd(dy2.data_ptr(), xs.data_ptr(), mean.data_ptr(), rstd.data_ptr(),
                                                   gamma.data_ptr(), _lib.ptr(dres), dx.data_ptr(), dg.data_ptr(),
                                                   db.data_ptr(), int(acc), sc.data_ptr(), M, H, _lib.cur_stream())
                _lib.check(rc, "cocclkLayerNormBwd")

            mg, mb = getattr(gamma, "main_grad", None), getattr(beta, "main_grad", None)
            if mg is not None and mb is not None:
                run(mg, mb, True)
                dgamma = dbeta = None
            else:
                dg = torch.empty(H, dtype=torch.float32, device=xs.device)
                db = torch.empty(H, dtype=torch.float32, device=xs.device)
                run(dg, db, False)
                dgamma, dbeta = dg.to(gamma.dtype), db.to(beta.dtype)
        else:
            xh = (xs.float() - mean[:, None]) * rstd[:, None]
            d = dy2.float()
            dyg = d * gamma.float()
            c1 = dyg.mean(-1, keepdim=True)
            c2 = (dyg * xh).mean(-1, keepdim=True)
            dxf = rstd[:, None] * (dyg - c1 - xh * c2)
            if dres is not None:
                dxf = dxf + dres.float()
            dx = dxf.to(xs.dtype)
            dg, db = (d * xh).sum(0), d.sum(0)
            dgamma = _cpu_param_grad(gamma, dg)
            dbeta = _cpu_param_grad(beta, db)
        dx = dx.reshape(ctx.shape)
        return dx, (dx if ctx.has_res else None), dgamma, dbeta, None


def _cpu_param_grad(p, g32):
    mg = getattr(p, "main_grad", None)
    if mg is not None:
        mg.add_(g32.reshape(mg.shape))
        return None
    return g32.to(p.dtype)


def layer_norm(x, gamma, beta, eps: float = 1e-5, residual=None):
    """y = LN(x + residual); returns (y, x + residual) when a residual is given, else y."""
    y, xs = _LayerNorm.apply(x, residual, gamma, beta, eps)
    return (y, xs) if residual is not None else y


# --------------------------------------------------------------------------- embeddings
class _Embed(torch.autograd.Function):
    @staticmethod
    def forward(ctx, wte, wpe, ids, first):
        b, s = ids.shape
        flat = ids.reshape(-1).contiguous()   # a column of a wider tensor is a strided view, and the kernels read consecutive ids
        e = F.embedding(flat, wte)
        if wpe is not None:
            e.view(b, s, -1).add_(wpe[first:first + s])
        ctx.save_for_backward(flat)
        # the tables' values are not needed again, only their gradient buffers: those of the parameters themselves, which a
        # saved-tensor hook would hand back as plain tensors
        ctx.tables = (wte, wpe)
        ctx.meta = (b, s, first)
        ctx.branch = Branch.current()
        return e

    @staticmethod
    def backward(ctx, dy):
        (flat,) = ctx.saved_tensors
        wte, wpe = ctx.tables
        b, s, first = ctx.meta
        T, H = b * s, wte.shape[1]
        (node_w, _), (node_p, _) = ctx.next_functions[:2]
        grads, straight = [None, None], []
        for i, (w, node) in enumerate(((wte, node_w), (wpe, node_p))):
            want = _wanted_gradient(w, node)
            straight.append(want == "buffer")
            if want == "tensor" and i == 0:
                grads[0] = torch.ops.aten.embedding_dense_backward(dy, flat, wte.shape[0], -1, False)
            elif want == "tensor":
                grads[1] = F.pad(dy.reshape(b, s, H).sum(0), (0, 0, first, wpe.shape[0] - first - s))
        if any(straight):
            dy = dy.contiguous() if aligned16(dy) else dy.clone(memory_format=torch.contiguous_format)
        lib = _lib.lib()
        sc = torch.empty(lib.cocclkEmbedScratchBytes(T, H), dtype=torch.uint8, device=dy.device) if straight[0] else None

        def into_buffers():
            st = _lib.cur_stream()
            if straight[0]:
                _lib.check(lib.cocclkEmbedBwd(dy.data_ptr(), flat.data_ptr(), sc.data_ptr(), wte.main_grad.data_ptr(), T, H,
                                              wte.shape[0], st), "cocclkEmbedBwd")
            if straight[1]:
                g = wpe.main_grad[first:first + s]
                _lib.check(lib.cocclkEmbedPositionsBwd(dy.data_ptr(), g.data_ptr(), b, s, H, st), "cocclkEmbedPositionsBwd")
        if ctx.branch is not None:   # behind the gradient of a tied output head, which goes into the same buffer
            ctx.branch.run(into_buffers, dy, flat, sc)
        else:
            into_buffers()
        return grads[0], grads[1], None, None


def _wanted_gradient(w, node) -> str:
    """How this backward pass wants the gradient of table `w` (`node`: where autograd would accumulate it): "buffer" (straight
    into `main_grad`), "tensor" (as a tensor: hooks on the table see and may change it, torch.autograd.grad returns it, a pass
    with create_graph differentiates it) or "none" (backward(inputs=...) of other tensors)."""
    if w is None or node is None:
        return "none"
    try:
        if not torch._C._will_engine_execute_node(node):
            return "none"
    except RuntimeError:   # a leaf whose gradient torch.autograd.grad captures
        return "tensor"
    return "tensor" if torch.is_grad_enabled() or w._backward_hooks or w._post_accumulate_grad_hooks else "buffer"


def embed_fits(ids, wte, wpe=None, first: int = 0) -> bool:
    """Whether the embedding gradient can go straight into the parameters' gradient buffers: bf16 tables on the GPU with fp32
    `main_grad` buffers, rows of whole 16-byte vectors, and at most 16384 tokens (the kernel that sorts them compares every
    pair: 72 us at that size; larger batches take PyTorch's gradient)."""
    def table(w):
        mg = getattr(w, "main_grad", None)
        return (w.is_cuda and w.dtype == torch.bfloat16 and w.dim() == 2 and w.is_contiguous() and w.shape[1] % 8 == 0 and
                w.requires_grad and mg is not None and mg.dtype == torch.float32 and mg.is_contiguous() and aligned16(mg))
    return (ordinary(ids, wte, wpe) and ids.is_cuda and ids.dtype == torch.int64 and ids.dim() == 2 and 0 < ids.numel() <= 16384 and table(wte) and
            (wpe is None or (table(wpe) and wpe.shape[1] == wte.shape[1] and wpe.shape[0] >= first + ids.shape[1])))


def embed(ids, wte, wpe=None, first: int = 0):
    """wte[ids] (+ wpe[first + position]) as [tokens, hidden] for ids [batch, seq]; the gradients are added to the tables'
    `main_grad` in fp32 (the caller has checked embed_fits), or handed to autograd where something wants to see them."""
    return _Embed.apply(wte, wpe, ids, first)


# The backward kernels' results are constants to autograd. Under create_graph (a backward pass with gradients enabled) the
# backward functions below are PyTorch operations instead, written out: their results can be differentiated again.
def _rms_norm_graph(x, weight, eps, dy):
    """(dx, dw) of RMSNorm(x) * weight; dw is None where it went into `main_grad`."""
    from ..models.llama import rms_norm_gradients
    rstd = torch.rsqrt(x.float().square().mean(-1, keepdim=True) + eps)
    dx, dw = rms_norm_gradients(x, weight, rstd, dy)
    mg = getattr(weight, "main_grad", None)
    if mg is not None:
        mg.add_(dw.detach())
        return dx, None
    return dx, dw.to(weight.dtype)


# --------------------------------------------------------------------------- RMSNorm (+ residual add)
class _RmsNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, res, weight, eps):
        H = x.shape[-1]
        xc = x.contiguous()
        r2 = res.contiguous() if res is not None else None
        y = torch.empty_like(xc)
        xo = torch.empty_like(xc) if res is not None else None
        M = x.numel() // H
        rstd = torch.empty(M, dtype=torch.float32, device=x.device)
        rc = _lib.lib().cocclkRmsNormFwd(xc.data_ptr(), _lib.ptr(r2), weight.data_ptr(), y.data_ptr(), _lib.ptr(xo),
                                         rstd.data_ptr(), M, H, eps, _lib.cur_stream())
        _lib.check(rc, "cocclkRmsNormFwd")
        ctx.save_for_backward(xo if res is not None else x, weight, rstd)
        ctx.has_res, ctx.eps = res is not None, eps
        return y, xo

    @staticmethod
    def backward(ctx, dy, dxs):
        xs, weight, rstd = ctx.saved_tensors
        if torch.is_grad_enabled():
            dx, dw = _rms_norm_graph(xs, weight, ctx.eps, dy)
            dx = dx + dxs if dxs is not None else dx
            return dx, (dx if ctx.has_res else None), dw, None
        xs = xs.contiguous()
        H = xs.shape[-1]
        M = xs.numel() // H
        dy2 = dy.reshape(-1, H).contiguous()
        dres = dxs.reshape(-1, H).contiguous() if dxs is not None else None
        if not (aligned16(dy2) and aligned16(dres)):
            dy2, dres = dy2.clone(), (dres.clone() if dres is not None else None)
        dx = torch.empty_like(xs)
        sc = scratch(xs.device, _lib.lib().cocclkLayerNormBwdGrid(M) * H, "ln")

        def run(out, acc):
            rc = _lib.lib().cocclkRmsNormBwd(dy2.data_ptr(), xs.data_ptr(), rstd.data_ptr(), weight.data_ptr(), _lib.ptr(dres),
                                             dx.data_ptr(), out.data_ptr(), int(acc), sc.data_ptr(), M, H, _lib.cur_stream())
            _lib.check(rc, "cocclkRmsNormBwd")

        dw = _accum_param_grad(weight, None, run)
        return dx, (dx if ctx.has_res else None), dw, None


def ordinary(*ts) -> bool:
    """Whether a kernel may stand in for PyTorch operations on these tensors (None counts): plain tensors, outside of function
    transforms (vmap, jvp, ...), forward-mode levels and dispatch modes (fake tensors, tracing, counters), all of which work on
    the operations and would not see a kernel."""
    return (all(t is None or type(t) in (torch.Tensor, torch.nn.Parameter) for t in ts) and
            not torch._C._are_functorch_transforms_active() and torch.autograd.forward_ad._current_level < 0 and
            torch._C._len_torch_dispatch_stack() == 0)


def aligned16(*ts) -> bool:
    """Whether every given tensor starts on a 16-byte boundary (None counts as aligned)."""
    return all(t is None or t.data_ptr() % 16 == 0 for t in ts)


def rms_norm_fits(x, weight, residual=None) -> bool:
    """Whether the RMSNorm kernel takes these tensors: bf16 on the GPU, rows of whole 16-byte vectors up to 16384 wide, fp32
    weight gradient. Everything else runs as PyTorch operations (models.llama.rms_norm)."""
    H = x.shape[-1] if x.dim() else 0
    same = residual is None or (residual.dtype == x.dtype and residual.shape == x.shape and residual.device == x.device)
    mg = getattr(weight, "main_grad", None)
    return (ordinary(x, weight, residual) and x.is_cuda and x.dtype == weight.dtype == torch.bfloat16 and weight.device == x.device and same and
            0 < H <= 16384 and H % 8 == 0 and x.numel() > 0 and weight.shape == (H,) and weight.is_contiguous() and
            (mg is None or (mg.dtype == torch.float32 and mg.is_contiguous())) and aligned16(x, weight, residual))


def rms_norm(x, weight, eps: float, residual=None):
    """y = RMSNorm(x + residual) * weight in one kernel; returns (y, x + residual) when a residual is given, else y."""
    y, xs = _RmsNorm.apply(x, residual, weight, eps)
    return (y, xs) if residual is not None else y


# --------------------------------------------------------------------------- rotation of queries and keys, SwiGLU gate
class _RotateQkv(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, qw, kw, cos, sin, nh, nkv, eps):
        T, d = qkv.shape[0], cos.shape[1]
        q = qkv.new_empty(T, nh, d)
        k, v = qkv.new_empty(T, nkv, d), qkv.new_empty(T, nkv, d)
        rc = _lib.lib().cocclkRotateFwd(qkv.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), cos.data_ptr(), sin.data_ptr(),
                                        _lib.ptr(qw), _lib.ptr(kw), T, cos.shape[0], nh, nkv, d, eps, _lib.cur_stream())
        _lib.check(rc, "cocclkRotateFwd")
        ctx.save_for_backward(qkv if qw is not None else None, qw, kw, cos, sin)
        ctx.meta = (nh, nkv, eps)
        return q, k, v

    @staticmethod
    def backward(ctx, dq, dk, dv):
        qkv, qw, kw, cos, sin = ctx.saved_tensors
        nh, nkv, eps = ctx.meta
        T, d = dq.shape[0], cos.shape[1]
        if torch.is_grad_enabled():
            return (*_rotate_graph(dq, dk, dv, qkv, qw, kw, cos, sin, eps), None, None, None, None, None)
        dq, dk, dv = (t.contiguous() if aligned16(t) else t.clone(memory_format=torch.contiguous_format) for t in (dq, dk, dv))
        dqkv = dq.new_empty(T, (nh + 2 * nkv) * d)
        mq, mk = getattr(qw, "main_grad", None), getattr(kw, "main_grad", None)
        sc = None
        if qw is not None:
            sc = scratch(dq.device, _lib.lib().cocclkRotateBwdGrid(T) * 2 * d, "rotate")
            if mq is None:
                gq, gk = (torch.empty(d, dtype=torch.float32, device=dq.device) for _ in range(2))
            else:
                gq, gk = mq, mk
        else:
            gq = gk = None
        rc = _lib.lib().cocclkRotateBwd(dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), _lib.ptr(qkv), dqkv.data_ptr(), cos.data_ptr(),
                                        sin.data_ptr(), _lib.ptr(qw), _lib.ptr(kw), _lib.ptr(gq), _lib.ptr(gk), int(mq is not None),
                                        _lib.ptr(sc), T, cos.shape[0], nh, nkv, d, eps, _lib.cur_stream())
        _lib.check(rc, "cocclkRotateBwd")
        if qw is not None and mq is None:
            return dqkv, gq.to(qw.dtype), gk.to(kw.dtype), None, None, None, None, None
        return dqkv, None, None, None, None, None, None, None


def _rotate_graph(dq, dk, dv, qkv, qw, kw, cos, sin, eps):
    """(dqkv, dqw, dkw) of the rotation under create_graph."""
    T, d = dq.shape[0], cos.shape[1]
    at = torch.arange(T, device=dq.device) % cos.shape[0]
    c, s = cos[at][:, None], sin[at][:, None]

    def back(g):   # the rotation by the opposite angle
        g = g.float()
        return g * c - torch.cat([-g[..., d // 2:], g[..., :d // 2]], -1) * s
    gq, gk = back(dq).to(dq.dtype), back(dk).to(dk.dtype)
    dqw = dkw = None
    if qw is not None:
        q, k, _ = (t.reshape(T, -1, d) for t in qkv.split([g.shape[1] * d for g in (dq, dk, dv)], -1))
        gq, dqw = _rms_norm_graph(q, qw, eps, gq)
        gk, dkw = _rms_norm_graph(k, kw, eps, gk)
    return torch.cat([t.reshape(T, -1) for t in (gq, gk, dv)], -1), dqw, dkw


def rotate_qkv_fits(qkv, d: int, qw=None, kw=None) -> bool:
    """Whether the rotation kernel takes a packed projection: contiguous bf16 on the GPU, heads of 32, 64, 128 or 256 (a head
    is a power of two of lanes), norm weights both present with fp32 gradients of the same kind, or both absent."""
    if not (ordinary(qkv, qw, kw) and qkv.is_cuda and qkv.dtype == torch.bfloat16 and qkv.dim() == 2 and qkv.is_contiguous() and qkv.numel() > 0 and
            d in (32, 64, 128, 256) and aligned16(qkv)):
        return False
    if qw is None and kw is None:
        return True
    if qw is None or kw is None:
        return False
    grads = [getattr(w, "main_grad", None) for w in (qw, kw)]
    return (all(w.dtype == torch.bfloat16 and w.shape == (d,) and w.is_contiguous() and w.device == qkv.device and aligned16(w)
                for w in (qw, kw)) and (grads[0] is None) == (grads[1] is None) and
            all(g is None or (g.dtype == torch.float32 and g.is_contiguous()) for g in grads))


def rotate_qkv(qkv, cos, sin, nh: int, nkv: int, qw=None, kw=None, eps: float = 1e-6):
    """qkv [tokens, (nh + 2 nkv) d] -> (q [tokens, nh, d], k, v [tokens, nkv, d]) with queries and keys normalised per head
    (qw, kw given) and rotated; cos / sin [seq, d] as the tables of models.llama, position = token % seq."""
    return _RotateQkv.apply(qkv, qw, kw, cos, sin, nh, nkv, eps)


class _Swiglu(torch.autograd.Function):
    @staticmethod
    def forward(ctx, z):
        F_ = z.shape[-1] // 2
        z2 = z.reshape(-1, 2 * F_)
        y = z2.new_empty(z2.shape[0], F_)
        _lib.check(_lib.lib().cocclkSwigluFwd(z2.data_ptr(), y.data_ptr(), z2.shape[0], F_, _lib.cur_stream()), "cocclkSwigluFwd")
        ctx.save_for_backward(z)
        return y.reshape(*z.shape[:-1], F_)

    @staticmethod
    def backward(ctx, dy):
        (z,) = ctx.saved_tensors
        if torch.is_grad_enabled():
            gate, up = z.chunk(2, dim=-1)
            return torch.autograd.grad(F.silu(gate) * up, z, dy, create_graph=True)[0]
        F_ = z.shape[-1] // 2
        dy = dy.contiguous() if aligned16(dy) else dy.clone(memory_format=torch.contiguous_format)
        dz = torch.empty_like(z)
        _lib.check(_lib.lib().cocclkSwigluBwd(dy.data_ptr(), z.data_ptr(), dz.data_ptr(), z.numel() // (2 * F_), F_,
                                              _lib.cur_stream()), "cocclkSwigluBwd")
        return dz


def swiglu(z):
    """silu(gate) * up for z = [gate | up] along the last dimension: one kernel each way for contiguous bf16 CUDA tensors
    whose halves are whole 16-byte vectors, PyTorch operations otherwise."""
    if (ordinary(z) and z.is_cuda and z.dtype == torch.bfloat16 and z.is_contiguous() and z.shape[-1] % 16 == 0 and z.numel() > 0 and
            aligned16(z)):
        return _Swiglu.apply(z)
    gate, up = z.chunk(2, dim=-1)
    return F.silu(gate) * up


# --------------------------------------------------------------------------- Linear (+bias, +GELU)
class _Linear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, bias, gelu):
        K = x.shape[-1]
        x2 = x.reshape(-1, K)
        N = w.shape[0]
        z = None
        if x.is_cuda:
            if gelu:
                y, z = G.gemm(x2, w, bias=bias, gelu=True, save_preact=True)
            else:
                y = G.gemm(x2, w, bias=bias)
        else:
            yf = x2.float() @ w.float().t()
            if bias is not None:
                yf = yf + bias.float()
            if gelu:
                z = yf.to(x.dtype)
                yf = F.gelu(z.float(), approximate="tanh")
            y = yf.to(x.dtype)
        ctx.save_for_backward(x2, w, bias if bias is not None else None, z)
        ctx.gelu = gelu
        ctx.has_bias = bias is not None
        ctx.in_shape = x.shape
        ctx.branch = Branch.current()
        return y.reshape(*x.shape[:-1], N)

    @staticmethod
    def backward(ctx, dy):
        x2, w, bias, z = ctx.saved_tensors
        N, K = w.shape
        dy2 = dy.reshape(-1, N)
        M = dy2.shape[0]
        if dy2.is_cuda:
            dy2 = dy2.contiguous()
            if ctx.gelu:
                dz = torch.empty_like(dy2)
                rc = _lib.lib().cocclkGeluBwd(dy2.data_ptr(), z.data_ptr(), dz.data_ptr(), dz.numel(), _lib.cur_stream())
                _lib.check(rc, "cocclkGeluBwd")
                dy2 = dz

            def parameter_grads():
                dw = _accum_param_grad(w, None, lambda out, acc: G.gemm(dy2.t(), x2.t(), out=out, accumulate=acc))
                db = None
                if ctx.has_bias:
                    def colsum(out, acc):
                        sc = scratch(dy2.device, _lib.lib().cocclkColSumBlocks(M) * N, "colsum")
                        rc = _lib.lib().cocclkColSum(dy2.data_ptr(), out.data_ptr(), int(acc), sc.data_ptr(), M, N,
                                                     _lib.cur_stream())
                        _lib.check(rc, "cocclkColSum")
                    db = _accum_param_grad(bias, None, colsum)
                return dw, db
            buffers = all(p is None or getattr(p, "main_grad", None) is not None for p in (w, bias))
            beside = ctx.branch is not None and buffers
            if beside:
                dw, db = ctx.branch.run(parameter_grads, dy2, x2)
            dx = G.gemm(dy2, w.t()) if ctx.needs_input_grad[0] else None
            if not beside:
                dw, db = parameter_grads()
        else:
            d = dy2.float()
            if ctx.gelu:
                zf = z.float().requires_grad_(True)
                with torch.enable_grad():
                    a = F.gelu(zf, approximate="tanh")
                d = torch.autograd.grad(a, zf, d)[0].to(dy.dtype).float()
            dx = (d @ w.float()).to(dy.dtype) if ctx.needs_input_grad[0] else None
            dw = _cpu_param_grad(w, d.t() @ x2.float())
            db = _cpu_param_grad(bias, d.sum(0)) if ctx.has_bias else None
        if dx is not None:
            dx = dx.reshape(ctx.in_shape)
        return dx, dw, db, None


def linear(x, w, bias=None, gelu: bool = False):
    """y = act(x @ w.T + bias); w is [out, in]; GELU (tanh form) fused into the GEMM epilogue."""
    return _Linear.apply(x, w, bias, gelu)


# --------------------------------------------------------------------------- cross-entropy
class _CrossEntropy(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, targets, scale, unit_grad):
        V = logits.shape[-1]
        lg = logits.reshape(-1, V)
        tg = targets.reshape(-1).contiguous()   # the kernel reads consecutive targets
        M = lg.shape[0]
        if lg.is_cuda:
            assert lg.stride(1) == 1
            loss = torch.empty(M, dtype=torch.float32, device=lg.device)
            rc = _lib.lib().cocclkCrossEntropy(lg.data_ptr(), tg.data_ptr(), loss.data_ptr(), M, V, lg.stride(0),
                                               float(scale), _lib.cur_stream())
            _lib.check(rc, "cocclkCrossEntropy")
            grad = lg  # overwritten in place with (softmax - onehot) * scale
        else:
            lf = lg.float()
            lse = torch.logsumexp(lf, -1)
            valid = tg >= 0
            tcl = tg.clamp(min=0)
            loss = torch.where(valid, lse - lf.gather(1, tcl[:, None])[:, 0], torch.zeros_like(lse))
            p = torch.softmax(lf, -1)
            p[torch.arange(M), tcl] -= 1.0
            p = p * valid[:, None]
            grad = (p * scale).to(lg.dtype)
        ctx.save_for_backward(grad)
        ctx.shape = logits.shape
        ctx.unit_grad = unit_grad
        return loss.sum() * scale

    @staticmethod
    def backward(ctx, dloss):
        (grad,) = ctx.saved_tensors
        if not ctx.unit_grad:
            grad = grad * dloss.to(grad.dtype)
        return grad.reshape(ctx.shape), None, None, None


def cross_entropy(logits, targets, scale: float, unit_grad: bool = True):
    """sum_i CE(logits_i, targets_i) * scale. On CUDA the logits buffer is consumed (turned into its gradient).

    unit_grad=True (the trainer's case) assumes the result is the root of backward(), i.e. the incoming
    gradient is 1, and skips one pass over the [tokens, vocab] gradient."""
    return _CrossEntropy.apply(logits, targets, scale, unit_grad)


# --------------------------------------------------------------------------- optimizer kernels
def adam_step(master, m, v, grad, param_bf16, *, lr, beta1, beta2, eps, weight_decay, step, grad_scale=None):
    n = master.numel()
    if master.is_cuda:
        rc = _lib.lib().cocclkAdam(master.data_ptr(), m.data_ptr(), v.data_ptr(), grad.data_ptr(),
                                   int(grad.dtype == torch.bfloat16), _lib.ptr(param_bf16), n, lr, beta1, beta2, eps,
                                   weight_decay, step, _lib.ptr(grad_scale), _lib.cur_stream())
        _lib.check(rc, "cocclkAdam")
        return
    g = grad.float() * (grad_scale.item() if grad_scale is not None else 1.0)
    m.mul_(beta1).add_(g, alpha=1 - beta1)
    v.mul_(beta2).addcmul_(g, g, value=1 - beta2)
    bc1, bc2 = 1 - beta1 ** step, 1 - beta2 ** step
    upd = (m / bc1) / ((v / bc2).sqrt() + eps) + weight_decay * master
    master.add_(upd, alpha=-lr)
    if param_bf16 is not None:
        param_bf16.copy_(master)


def sum_squares(x, out, accumulate=False):
    """out[0] (+)= sum(x^2) without a host sync."""
    if x.is_cuda:
        sc = scratch(x.device, _lib.lib().cocclkSumSqBlocks(x.numel()), "sumsq")
        rc = _lib.lib().cocclkSumSq(x.data_ptr(), int(x.dtype == torch.bfloat16), x.numel(), out.data_ptr(),
                                    int(accumulate), sc.data_ptr(), _lib.cur_stream())
        _lib.check(rc, "cocclkSumSq")
    else:
        s = x.float().pow(2).sum()
        out[0] = out[0] + s if accumulate else s


def clip_coef(sumsq, max_norm: float, grad_scale_in: float, coef, norm_out=None):
    if sumsq.is_cuda:
        rc = _lib.lib().cocclkClipCoef(sumsq.data_ptr(), max_norm, grad_scale_in, coef.data_ptr(), _lib.ptr(norm_out),
                                       _lib.cur_stream())
        _lib.check(rc, "cocclkClipCoef")
    else:
        norm = sumsq[0].sqrt() * grad_scale_in
        if norm_out is not None:
            norm_out[0] = norm
        c = 1.0
        if max_norm > 0 and norm > max_norm:
            c = max_norm / (norm + 1e-6)
        coef[0] = c * grad_scale_in

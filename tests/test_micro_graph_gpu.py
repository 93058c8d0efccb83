"""The replayed micro-batch of small models against the launched one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cfg(arch):
    from coccl_b200.models.gpt import GPTConfig
    if arch == "gpt":
        return GPTConfig(n_layer=2, hidden=256, n_head=4, ffn=1024, seq_len=96, vocab=1024)
    return GPTConfig(arch="llama", n_layer=2, hidden=256, n_head=4, n_kv_head=2, ffn=512, seq_len=96, vocab=1024, qkv_bias=True,
                     qk_norm=True, tie_embeddings=False, rope_theta=1.0e4)


def _pair(arch):
    from coccl_b200.train import Trainer
    dev = torch.device("cuda", 0)
    out = [Trainer(_cfg(arch), dev, micro_batch=2, lr=1e-3, seed=5) for _ in range(2)]
    out[1].micro_graph.enabled = False
    return out


def _tokens(seed, n=4, seq=96):
    return torch.randint(0, 1024, (n, seq + 1), generator=torch.Generator().manual_seed(seed)).pin_memory()


@pytest.mark.parametrize("arch", ["gpt", "llama"])
def test_replayed_steps_equal_launched_steps(cuda, arch):
    """New tokens every step, a buffer of the trainer's scratch replaced by a larger one in between, another number of
    micro-batches and another sequence length: same losses and gradients up to the order of the attention's atomic sums."""
    from coccl_b200.ops import fused
    a, b = _pair(arch)
    for step in range(8):
        if step == 5:
            for (index, tag), t in list(fused._scratch.items()):
                fused.scratch(torch.device("cuda", index), 2 * t.numel(), tag).fill_(float("nan"))
        tok = _tokens(step, 8 if step == 6 else 4, 64 if step == 7 else 96)
        la, lb = a.train_step(tok).item(), b.train_step(tok).item()
        assert abs(la - lb) <= 2e-3 * abs(lb), (step, la, lb)
        ga, gb = a.stage.store.flat_grad, b.stage.store.flat_grad
        assert (ga - gb).norm() <= 2e-2 * gb.norm(), step
        assert (a.micro_graph.graph is not None) == (2 <= step <= 5), step
    a.check_health()


def test_hooks_modes_and_changed_buffers_take_the_launches(cuda):
    a, _ = _pair("gpt")
    tok = _tokens(1)
    for _ in range(3):
        a.train_step(tok)
    assert a.micro_graph.graph is not None
    seen = []
    h = a.stage.layers[0].register_forward_hook(lambda *x: seen.append(1))
    a.train_step(tok)
    assert len(seen) == 2
    h.remove()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(2), t)[1], lambda t: t):
        a.train_step(tok)
    assert seen.count(2) > 0
    a.train_step(tok)
    assert a.micro_graph.graph is not None
    p = a.stage.layers[0].qkv_weight
    p.main_grad = p.main_grad.clone()      # another gradient buffer: the captured one must not be written instead
    a.train_step(tok)
    assert a.micro_graph.graph is None and float(p.main_grad.norm()) > 0


def _set(obj, name, value):
    setattr(obj, name, value)


def _other_data(p):
    p.data = (p.data.float() * 0.5).to(p.dtype)   # another buffer


def _other_main_grad(p):
    p.main_grad = p.main_grad.clone()


def _plain_mlp(t):
    layer = t.stage.layers[0]
    layer.mlp = lambda y: type(layer).mlp(layer, y) * 0.5


CHANGES = {
    "weight of the joined projections": lambda t: _other_data(t.stage.layers[0].wqkv),
    "weight of gate and up": lambda t: _other_data(t.stage.layers[1].w_gate_up),
    "gradient buffer of the joined projections": lambda t: _other_main_grad(t.stage.layers[0].wqkv),
    "eps": lambda t: _set(t.cfg, "eps", 0.5),
    "rope_theta": lambda t: _set(t.cfg, "rope_theta", 7.0),
    "method of a layer": _plain_mlp,
}


@pytest.mark.parametrize("change", sorted(CHANGES))
def test_changes_after_the_capture_take_effect(cuda, change):
    """The same change made to a replayed and to a launched trainer: their next steps agree up to the order of the attention's
    atomic sums, and differ from what a step without the change gives."""
    a, b = _pair("llama")
    for step in range(4):
        a.train_step(_tokens(step))
        b.train_step(_tokens(step))
    assert a.micro_graph.graph is not None
    for t in (a, b):
        CHANGES[change](t)
    for step in range(4, 8):
        la, lb = a.train_step(_tokens(step)).item(), b.train_step(_tokens(step)).item()
        assert abs(la - lb) <= 2e-3 * abs(lb), (step, la, lb)
        for pa, pb in zip(a.stage.parameters(), b.stage.parameters()):
            assert (pa.main_grad - pb.main_grad).norm() <= 3e-2 * pb.main_grad.norm() + 1e-6, step
    assert (a.micro_graph.graph is not None) == (change != "method of a layer")   # captured anew, or not at all


@pytest.mark.parametrize("switch", ["attention kernels", "determinism"])
def test_switches_of_pytorch_send_the_step_back_to_the_launches(cuda, switch):
    from torch.nn.attention import SDPBackend, sdpa_kernel
    a, _ = _pair("gpt")
    for step in range(3):
        a.train_step(_tokens(step))
    graph = a.micro_graph.graph
    assert graph is not None
    if switch == "attention kernels":
        with sdpa_kernel(SDPBackend.MATH):
            a.train_step(_tokens(3))
    else:
        torch.use_deterministic_algorithms(True, warn_only=True)
        try:
            a.train_step(_tokens(3))
        finally:
            torch.use_deterministic_algorithms(False)
    assert a.micro_graph.graph is None


def test_disabling_gives_the_graph_back(cuda):
    a, b = _pair("gpt")
    for step in range(3):
        a.train_step(_tokens(step))
        b.train_step(_tokens(step))
    assert a.micro_graph.graph is not None
    a.micro_graph.enabled = False
    la, lb = a.train_step(_tokens(3)).item(), b.train_step(_tokens(3)).item()
    assert a.micro_graph.graph is None and abs(la - lb) <= 2e-3 * abs(lb)


def test_failed_capture_is_reported_and_the_launches_take_over(cuda, monkeypatch):
    a, b = _pair("gpt")

    class Graph(torch.cuda.CUDAGraph):
        def capture_begin(self, *args, **kw):
            raise RuntimeError("no graph today")
    for step in range(5):
        with monkeypatch.context() as m:
            m.setattr(torch.cuda, "CUDAGraph", Graph)
            if step == 2:
                with pytest.warns(UserWarning, match="no graph today"):
                    la = a.train_step(_tokens(step)).item()
            else:
                la = a.train_step(_tokens(step)).item()
        lb = b.train_step(_tokens(step)).item()
        assert abs(la - lb) <= 2e-3 * abs(lb), step
    assert a.micro_graph.graph is None and not a.micro_graph.enabled


def test_gradients_that_autograd_hands_over_are_not_left_to_a_capture(cuda):
    """An embedding whose gradient buffer the kernels do not take gets its gradient through `.grad`."""
    a, b = _pair("llama")
    for t in (a, b):
        n = t.stage.wte.numel()
        t.stage.wte.main_grad = torch.zeros(n + 1, device=cuda)[1:].view_as(t.stage.wte)
    for step in range(5):
        for t in (a, b):
            t.stage.wte.main_grad.zero_()
        if step == 2:
            with pytest.warns(UserWarning, match="gradient"):
                a.train_step(_tokens(step))
        else:
            a.train_step(_tokens(step))
        b.train_step(_tokens(step))
        ga, gb = a.stage.wte.main_grad, b.stage.wte.main_grad
        assert gb.norm() > 0 and (ga - gb).norm() <= 3e-2 * gb.norm(), step
    assert a.micro_graph.graph is None


@pytest.mark.parametrize("arch", ["gpt", "llama"])
def test_every_gradient_of_a_replayed_step(cuda, arch):
    """Parameter by parameter, from equal parameters: what the backward pass forms ahead of its first attention (head, last norm, the
    last layer's second half) bit for bit, the others up to the order of the attention's atomic sums."""
    a, b = _pair(arch)
    for step in range(5):
        a.stage.store.flat_param.copy_(b.stage.store.flat_param)
        a.train_step(_tokens(step))
        b.train_step(_tokens(step))
        if step < 2:
            continue
        assert a.micro_graph.graph is not None
        ours = dict(a.stage.named_parameters())
        for name, p in b.stage.named_parameters():
            got, want = ours[name].main_grad, p.main_grad
            assert want.norm() > 0, name
            if name.startswith(("lnf", "lm_head", "layers.1.fc", "layers.1.gate", "layers.1.up", "layers.1.w_gate", "layers.1.down", "layers.1.ln2")):
                assert torch.equal(got, want), (step, name)
            else:
                assert (got - want).norm() <= 2e-2 * want.norm(), (step, name)


def test_a_bound_on_the_pool_leaves_the_branch_out(cuda, monkeypatch):
    """Between the two sizes of the pool the graph is captured in one stream, with the same gradients."""
    from coccl_b200.ops import fused
    from coccl_b200.train import MicroBatchGraph
    a, b = _pair("gpt")
    n = 2 * 96
    small, large = (MicroBatchGraph.pool_bytes(a.cfg, n, branch) for branch in (False, True))
    monkeypatch.setattr(MicroBatchGraph, "MAX_POOL_BYTES", (small + large) // 2)
    made = []
    init = fused.Branch.__init__

    def counted(self, device):
        made.append(device)
        init(self, device)
    monkeypatch.setattr(fused.Branch, "__init__", counted)
    for bound, branches in (((small + large) // 2, 0), (large, 1)):
        monkeypatch.setattr(MicroBatchGraph, "MAX_POOL_BYTES", bound)
        a.micro_graph._drop()
        for step in range(3):
            a.stage.store.flat_param.copy_(b.stage.store.flat_param)
            a.train_step(_tokens(step))
            b.train_step(_tokens(step))
        assert a.micro_graph.graph is not None and len(made) == branches
        ga, gb = a.stage.store.flat_grad, b.stage.store.flat_grad
        assert (ga - gb).norm() <= 2e-2 * gb.norm()


def test_an_error_inside_a_captured_pass_reaches_the_caller(cuda):
    """On the host, behind work of the gradients' branch; the next steps are launched and captured as if nothing had been."""
    from coccl_b200.ops import fused
    from coccl_b200.train import Trainer
    a, b = _pair("gpt")

    def fail(tokens, scale):
        Trainer._micro_batch(a, tokens, scale)
        assert fused.Branch.current().used
        raise ValueError("inside the pass")
    for step in range(5):
        if step == 2:
            a._micro_batch = fail
            with pytest.raises(ValueError, match="inside the pass"):
                a.micro_graph._capture(a, (2, 97), 1.0)
            del a._micro_batch
            assert a.micro_graph.graph is None and a.micro_graph.enabled
        la, lb = a.train_step(_tokens(step)).item(), b.train_step(_tokens(step)).item()
        assert abs(la - lb) <= 2e-3 * abs(lb), step
    assert a.micro_graph.graph is not None
    a.check_health()

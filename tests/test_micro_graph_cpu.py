"""The replay rule leaves CPU trainers alone, however the device is named."""
import pytest
import torch


def test_device_given_as_text():
    from coccl_b200.models.gpt import GPTConfig
    from coccl_b200.train import Trainer
    cfg = GPTConfig(n_layer=1, hidden=32, n_head=2, ffn=64, seq_len=8, vocab=64, dtype=torch.float32)
    tok = torch.randint(0, cfg.vocab, (2, cfg.seq_len + 1), generator=torch.Generator().manual_seed(3))
    by_text, by_device = Trainer(cfg, "cpu", micro_batch=2), Trainer(cfg, torch.device("cpu"), micro_batch=2)
    for _ in range(4):
        assert by_text.train_step(tok).item() == by_device.train_step(tok).item()
    assert by_text.micro_graph.graph is None and by_device.micro_graph.graph is None


def _trainer(arch="gpt"):
    from coccl_b200.models.gpt import GPTConfig
    from coccl_b200.train import Trainer
    extra = dict(n_kv_head=1, qkv_bias=True, qk_norm=True, tie_embeddings=False) if arch == "llama" else {}
    cfg = GPTConfig(arch=arch, n_layer=2, hidden=32, n_head=2, ffn=64, seq_len=8, vocab=64, dtype=torch.float32, **extra)
    return Trainer(cfg, "cpu", micro_batch=2)


def _replace_layer(t):
    t.stage.layers[1] = type(t.stage.layers[1]).__new__(type(t.stage.layers[1]))


CHANGES = {
    "field of the configuration": lambda t: setattr(t.cfg, "eps", 1e-3),
    "another configuration": lambda t: setattr(t.stage, "cfg", type(t.cfg)()),
    "attribute of a layer": lambda t: setattr(t.stage.layers[1], "idx", "one"),
    "layer": _replace_layer,
    "layer in the list of chunks": lambda t: t.stage.chunks[0].reverse(),
    "parameter": lambda t: setattr(t.stage.layers[0], "ln1_weight", torch.nn.Parameter(t.stage.layers[0].ln1_weight.data)),
    "object in an attribute": lambda t: setattr(t.stage.tp, "extra", 1),
    "stage": lambda t: setattr(t, "stage", _trainer().stage),
}


@pytest.mark.parametrize("arch", ["gpt", "llama"])
@pytest.mark.parametrize("change", sorted(CHANGES))
def test_snapshot_notices_what_a_pass_would_have_looked_up(arch, change):
    from coccl_b200.train import _Snapshot
    t = _trainer(arch)
    s = _Snapshot(t.stage, t.cfg)
    tok = torch.randint(0, 64, (2, 9), generator=torch.Generator().manual_seed(3))
    t.train_step(tok)
    handle = t.stage.layers[0].register_forward_hook(lambda *a: None)
    handle.remove()
    assert s.holds(t.stage, t.cfg)   # training itself, and a hook that is gone, change nothing
    CHANGES[change](t)
    assert not s.holds(t.stage, t.cfg)


@pytest.mark.parametrize("arch", ["gpt", "llama"])
def test_only_the_package_s_own_code_is_replayed(arch, monkeypatch):
    from coccl_b200.ops import fused
    from coccl_b200.train import MicroBatchGraph
    from coccl_b200.train import _own_code_in_place as unchanged
    own = MicroBatchGraph.own_code
    assert own(_trainer(arch).stage) and unchanged()
    t = _trainer(arch)
    t.stage.layers[0].forward = lambda *a: a
    assert not own(t.stage)
    t = _trainer(arch)
    t.stage.layers[1].mlp = lambda y: y
    assert not own(t.stage)
    t = _trainer(arch)
    t.stage.layers[1].__class__ = type("Other", (type(t.stage.layers[1]),), {})
    assert not own(t.stage)
    t = _trainer(arch)
    t.stage.layers[0].tp.linear_scatter = lambda x, w, bias=None: x
    assert not own(t.stage)
    t = _trainer(arch)
    t.stage.layers[0].tp = type("Other", (type(t.stage.tp),), {})()
    assert not own(t.stage)
    t = _trainer(arch)
    t.stage.extra = torch.nn.Linear(2, 2)
    assert not own(t.stage)
    for space, name in ((fused, "layer_norm"), (fused, "swiglu"), (type(t.stage), "embed"), (torch.nn.functional, "embedding")):
        with monkeypatch.context() as m:
            m.setattr(space, name, lambda *a, **k: None)
            assert not unchanged()
    assert unchanged()


def test_size_rule_counts_what_the_graph_would_keep():
    from coccl_b200.models.gpt import GPTConfig
    from coccl_b200.train import MicroBatchGraph
    small = dict(n_layer=2, hidden=256, n_head=4, ffn=1024, seq_len=2048)
    assert MicroBatchGraph.worth_it(GPTConfig(vocab=1024, **small), 8192)
    assert MicroBatchGraph.worth_it(GPTConfig(vocab=50304, **small), 8192)
    assert not MicroBatchGraph.worth_it(GPTConfig(vocab=50304, **small), 16384)   # 1.6 GB of logits


def test_size_rule():
    from coccl_b200.models.gpt import GPTConfig
    from coccl_b200.train import MicroBatchGraph
    small = GPTConfig(n_layer=2, hidden=256, n_head=4, ffn=1024, seq_len=96, vocab=1024)
    assert MicroBatchGraph.worth_it(small, 192)
    assert not MicroBatchGraph.worth_it(small, 16385)
    assert not MicroBatchGraph.worth_it(GPTConfig(), 4096)


class _Streams:
    """Streams, events and captures of torch.cuda as far as a capture sees them: a stream that has waited for one in a capture is in
    it too, and has to come back to the stream that the capture began in before that can end."""

    def __init__(self, monkeypatch):
        outer = self
        self.current, self.away, self.origin, self.ended = None, set(), None, 0

        class Stream:
            def __init__(self, device=None):
                self.device = device

            def wait_stream(self, other):
                if other is outer.origin or other in outer.away:
                    outer.away.add(self)
                if self is outer.origin:
                    outer.away.discard(other)
                    outer.away.discard(self)

        class use:
            def __init__(self, stream):
                self.stream = stream

            def __enter__(self):
                self.before, outer.current = outer.current, self.stream

            def __exit__(self, *_):
                outer.current = self.before

        class Graph:
            def capture_begin(self, **_):
                outer.origin = outer.current

            def capture_end(self):
                outer.origin = None
                outer.ended += 1
                if outer.away:
                    raise RuntimeError("capture ended with a stream that has not joined")

        self.current = Stream()
        for name, fake in (("Stream", Stream), ("stream", use), ("CUDAGraph", Graph), ("current_stream", lambda device=None: outer.current)):
            monkeypatch.setattr(torch.cuda, name, fake)


@pytest.mark.parametrize("error", [ValueError("in the pass"), KeyboardInterrupt("in the pass"), None], ids=["error", "interrupt", "none"])
@pytest.mark.parametrize("in_branch", [False, True])
def test_an_error_inside_a_captured_pass_stays_that_error(monkeypatch, error, in_branch):
    """The branch of parameter gradients joins whatever happens, so that the capture can be ended and what the caller sees is what went
    wrong."""
    from coccl_b200.ops import fused
    t = _trainer()
    streams = _Streams(monkeypatch)

    def fail():
        if error is not None:
            raise error

    def micro_batch(tokens, scale):
        branch = fused.Branch.current()
        branch.run(lambda: None, tokens)
        if in_branch:
            branch.run(fail, tokens)
        fail()
    monkeypatch.setattr(t, "_micro_batch", micro_batch, raising=False)
    if error is None:
        t.micro_graph._capture(t, (2, 9), 1.0)
    else:
        with pytest.raises(type(error), match="in the pass"):
            t.micro_graph._capture(t, (2, 9), 1.0)
    assert (t.micro_graph.graph is not None) == (error is None)
    assert streams.ended == 1 and not streams.away and fused.Branch.current() is None and t.micro_graph.enabled


def test_a_broken_capture_is_reported_with_its_own_error(monkeypatch):
    """An error that also breaks the capture: the streams can neither join nor end, and that is what is reported, as ever."""
    from coccl_b200.ops import fused
    t = _trainer()
    streams = _Streams(monkeypatch)

    def micro_batch(tokens, scale):
        branch = fused.Branch.current()
        branch.run(lambda: None, tokens)

        def broken(stream):
            raise RuntimeError("cannot join")
        monkeypatch.setattr(branch, "join", broken)
        raise RuntimeError("out of memory")
    monkeypatch.setattr(t, "_micro_batch", micro_batch, raising=False)
    with pytest.warns(UserWarning, match="not joined"):
        t.micro_graph._capture(t, (2, 9), 1.0)
    assert streams.ended == 1 and t.micro_graph.graph is None and not t.micro_graph.enabled

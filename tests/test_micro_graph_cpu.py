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

"""What a codec configuration keeps for its calls stays out of its identity."""
import copy
import dataclasses
import pickle

import pytest
import torch

from coccl_b200.ops.codec import CodecConfig


def test_layouts_are_no_part_of_a_configuration():
    a, b = CodecConfig("sdp4bit", 4, 128, False, True, seed=7), CodecConfig("sdp4bit", 4, 128, False, True, seed=7)
    n32, n16 = a.encoded_chunk_bytes(1000, torch.float32), a.encoded_chunk_bytes(1000, torch.bfloat16)
    assert (n32, n16) == (8 * 64 + 8 * 4, 8 * 64 + 8 * 8)
    assert a == b and hash(a) == hash(b) and repr(a) == repr(b) and dataclasses.asdict(a) == dataclasses.asdict(b)
    for c in (copy.copy(a), copy.deepcopy(a), pickle.loads(pickle.dumps(a))):
        assert c == a and "_layouts" not in vars(c)
        assert c.encoded_chunk_bytes(1000, torch.float32) == n32
    wider = dataclasses.replace(a, group=64)
    assert wider.encoded_chunk_bytes(1000, torch.float32) == 16 * 32 + 16 * 4
    assert a.layout(torch.float32)[0].paramBytes == 4 and a.layout(torch.float16)[0].paramBytes == 8
    assert a.layout(torch.float32)[0].seed == 7


def test_encoded_sizes_of_every_kind():
    want = {("zfp", 4): 500, ("zfp", 16): 2000, ("mxfp8", 8): 1024 + 32, ("taco", 8): 8 * 128 + 8 * 8}
    for (kind, bits), n in want.items():
        cfg = CodecConfig(kind, bits, {"zfp": 4, "mxfp8": 32, "taco": 128}[kind], False, False)
        assert cfg.encoded_chunk_bytes(1000, torch.float32) == n
    assert CodecConfig("zfp", 5, 4, False, False).encoded_chunk_bytes(1002, torch.float32) == -(-(251 * 20 // 8) // 4) * 4


def test_calls_leave_a_configuration_s_fields_alone():
    """`vars` are the fields, before and after a call: they build an equal configuration, and snapshots of them stay equal."""
    cfg = CodecConfig("taco", 8, 64, False, False)
    before = dict(vars(cfg))
    cfg.encoded_chunk_bytes(1000, torch.float32)
    assert vars(cfg) == before == dataclasses.asdict(cfg)
    assert CodecConfig(**vars(cfg)) == cfg
    assert cfg.layout(torch.float32)[0] is cfg.layout(torch.float32)[0]


def test_a_type_that_the_kernels_do_not_know_is_a_key_error(monkeypatch):
    """As a look-up of the type gives it, before anything is launched; sizes are known for every type."""
    from coccl_b200 import _lib
    from coccl_b200.ops import codec as C
    monkeypatch.setattr(_lib, "lib", lambda: type("", (), {"__getattr__": lambda self, name: lambda *a: 1 / 0})())
    monkeypatch.setattr(_lib, "cur_stream", lambda: 0)

    class OnGpu(torch.Tensor):
        is_cuda = True
    x = torch.zeros(256, dtype=torch.float64).as_subclass(OnGpu)
    enc = torch.zeros(1, 144, dtype=torch.uint8).as_subclass(OnGpu)
    assert C.SDP4BIT_G128.encoded_chunk_bytes(256, torch.float64) == 128 + 2 * 8
    with pytest.raises(KeyError):
        C.encode(x, C.SDP4BIT_G128, 1)
    with pytest.raises(KeyError):
        C.decode(enc, C.SDP4BIT_G128, 256, torch.float64, 1)

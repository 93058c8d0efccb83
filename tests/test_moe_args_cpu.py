"""Routing tables of different sizes before the expert exchange (the kernel library recorded in its place, no GPU)."""
import pytest
import torch

from coccl_b200 import _lib
from coccl_b200.ops import moe as MO


class _Recorder:
    def __init__(self, real):
        self.real, self.launched = real, []

    def cocclkMoeLayoutRanks(self, args, stream):
        self.launched.append("layout")
        return 0

    def cocclkMoeDispatch(self, args, ranks, max_ctas, stream):
        self.launched.append("dispatch")
        return 0

    def __getattr__(self, name):
        return getattr(self.real, name)


@pytest.fixture
def recorder(monkeypatch):
    rec = _Recorder(_lib.lib())
    monkeypatch.setattr(_lib, "lib", lambda: rec)
    monkeypatch.setattr(_lib, "cur_stream", lambda: 0)
    return rec


def _case(n=3, tokens=5, topk=2, hidden=16):
    return ([torch.zeros(tokens, hidden, dtype=torch.bfloat16) for _ in range(n)],
            [torch.zeros(tokens, topk, dtype=torch.int32) for _ in range(n)])


@pytest.mark.parametrize("shape", [(4, 2), (5, 1)])
@pytest.mark.parametrize("rank", [1, 2])
def test_shorter_tables_are_refused(recorder, rank, shape):
    """The layout of every rank has the entries of the first: a shorter table would be read, and its positions written, out of range."""
    xs, ids = _case()
    ids[rank] = torch.zeros(shape, dtype=torch.int32)
    with pytest.raises(ValueError):
        MO.emulate_dispatch(xs, ids, 6)
    assert not recorder.launched


@pytest.mark.parametrize("shape", [(6, 2), (5, 3)])
def test_longer_tables_have_layouts_of_their_own(recorder, shape):
    xs, ids = _case()
    ids[2] = torch.ones(shape, dtype=torch.int32)
    _, handles, _ = MO.emulate_dispatch(xs, ids, 6)
    assert recorder.launched == ["dispatch"]
    for h, i in zip(handles, ids):
        assert torch.equal(h.pos, MO.route_layout(i, 6, 3)[0])


def test_tables_of_one_size_and_any_stride_share_a_launch(recorder):
    xs, ids = _case()
    ids[1] = torch.zeros(2, 5, dtype=torch.int32).t()
    ids[2] = torch.zeros(10, dtype=torch.int32)   # as many entries in another shape: taken in their order, as ever
    MO.emulate_dispatch(xs, ids, 6)
    assert recorder.launched == ["layout", "dispatch"]

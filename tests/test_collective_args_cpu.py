"""The arguments that `emulate_collective` hands to the kernel library, recorded in its place (no GPU): every rank's entries are
filled, or the call is refused before anything is launched."""
import ctypes

import pytest
import torch

from coccl_b200 import _lib
from coccl_b200.ops import codec as C, collective as K


class _Recorder:
    """The kernel library's sizes, with launches kept instead of made."""

    def __init__(self, real):
        self.real, self.launched = real, []

    def cocclkFusedCollective(self, args, ranks, max_ctas, stream):
        kept = _lib.CollArgs()
        ctypes.memmove(ctypes.byref(kept), ctypes.byref(args), ctypes.sizeof(kept))
        self.launched.append((kept, ranks))
        return 0

    def __getattr__(self, name):
        return getattr(self.real, name)


@pytest.fixture
def recorder(monkeypatch):
    rec = _Recorder(_lib.lib())
    monkeypatch.setattr(_lib, "lib", lambda: rec)
    monkeypatch.setattr(_lib, "cur_stream", lambda: 0)
    return rec


def _inputs(n, numel=64 * 8):
    return [torch.zeros(numel) for _ in range(n)]


def _pointers(args, n):
    return [[getattr(args, f)[r] for r in range(n)] for f in ("inp", "out", "ws", "flags", "status")]


def test_a_state_of_fewer_ranks_is_refused_before_the_launch(recorder):
    state = {}
    K.emulate_collective("reduce_scatter", _inputs(2), C.SDP4BIT_G128, state=state)
    with pytest.raises(IndexError):
        K.emulate_collective("reduce_scatter", _inputs(4), C.SDP4BIT_G128, state=state)
    assert [ranks for _, ranks in recorder.launched] == [2]
    # the state still serves the ranks that it has buffers for
    K.emulate_collective("reduce_scatter", _inputs(2), C.SDP4BIT_G128, state=state)
    assert [ranks for _, ranks in recorder.launched] == [2, 2]


def test_a_state_of_more_ranks_serves_fewer(recorder):
    state = {}
    for n in (4, 2, 4):
        K.emulate_collective("all_gather", _inputs(n), C.SDP4BIT_G128, state=state)
        args, ranks = recorder.launched[-1]
        assert ranks == n and all(p is not None for row in _pointers(args, n) for p in row)


def test_delta_gather_with_fewer_outputs_than_ranks_is_refused(recorder):
    state = {"outs": [torch.zeros(4 * 512) for _ in range(3)]}
    with pytest.raises(IndexError):
        K.emulate_collective("all_gather_delta", _inputs(4), C.SDP4BIT_G128, state=state)
    assert not recorder.launched


@pytest.mark.parametrize("bad", [torch.zeros(64 * 8, 2)[:, 0], torch.zeros(64 * 8 - 1)], ids=["strided", "short"])
def test_every_rank_s_input_is_looked_at(recorder, bad):
    xs = _inputs(4)
    xs[3] = bad
    state = {}
    K.emulate_collective("reduce_scatter", _inputs(4), C.SDP4BIT_G128, state=state)
    with pytest.raises(AssertionError):
        K.emulate_collective("reduce_scatter", xs, C.SDP4BIT_G128, state=state)
    assert len(recorder.launched) == 1


@pytest.mark.parametrize("missing", ["inp", "out", "ws", "flags"])
@pytest.mark.parametrize("rank", [0, 3])
def test_the_library_refuses_arguments_without_a_buffer(recorder, missing, rank):
    """Checked before any call of the CUDA runtime, so it can be seen without a GPU."""
    K.emulate_collective("reduce_scatter", _inputs(4), C.SDP4BIT_G128)
    args, ranks = recorder.launched[-1]
    getattr(args, missing)[rank] = None
    assert recorder.real.cocclkFusedCollective(args, ranks, 0, None) == -1


def test_every_rank_s_result_is_a_tensor_of_its_own(recorder):
    """Of its own memory (kept, saved or resized by itself) and no view, which autograd would not let a caller change in place."""
    outs = K.emulate_collective("all_gather", _inputs(4, 1003), C.SDP4BIT_G128)
    assert all(o._base is None and o.is_contiguous() and o.storage_offset() == 0 and o.untyped_storage().nbytes() == o.nbytes for o in outs)
    outs[1].zero_()
    outs[0].resize_(2 * outs[0].numel()).fill_(7.0)
    assert not outs[1].any()
    outs[2].mul_(torch.ones_like(outs[2], requires_grad=True))
    assert outs[2].requires_grad

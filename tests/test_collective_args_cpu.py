"""The arguments that `emulate_collective` hands to the kernel library, recorded in its place (no GPU): every rank's entries are
filled, or the call is refused before anything is launched."""
import copy
import ctypes
import io

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


def test_a_state_can_be_copied_and_saved(recorder):
    """It holds buffers and their sizes, which a program may keep with its checkpoints; a copy serves as well as the original."""
    state = {}
    K.emulate_collective("reduce_scatter", _inputs(4), C.SDP4BIT_G128, state=state)
    assert set(state) == {"flags", "status", "ws", "ws_bytes"}
    file = io.BytesIO()
    torch.save(state, file)
    file.seek(0)
    for other in (copy.deepcopy(state), torch.load(file, weights_only=True)):
        K.emulate_collective("reduce_scatter", _inputs(4), C.SDP4BIT_G128, state=other)
        args, _ = recorder.launched[-1]
        assert args.ws[3] == other["ws"][3].data_ptr() != state["ws"][3].data_ptr()


def test_kinds_in_turn_and_what_they_share(recorder):
    """A call's own values (buffers, epoch, time limit, trace) are in its own arguments only."""
    kinds = [("reduce_scatter", 4, 64 * 8, C.SDP4BIT_G128, None), ("all_gather", 2, 64, C.MXFP8, 3), ("reduce_scatter", 4, 64 * 8, C.TACO_G128, None)]
    state, first = {}, []
    for turn in range(2):
        for i, (op, n, numel, cfg, tiles) in enumerate(kinds):
            if turn == 0 and i == 0:
                state["trace"] = [torch.zeros(8, dtype=torch.int64) for _ in range(4)]
            xs = _inputs(n, numel)
            outs = K.emulate_collective(op, xs, cfg, slice_tiles=tiles, epoch=1 + turn, timeout_ms=5.0 + i, state=state)
            state.pop("trace", None)
            a, ranks = recorder.launched[-1]
            alone = K._arguments(K.OP_NAMES[op], n, xs[0].dtype, numel, tiles, None, cfg)[0]
            for field in ("op", "nRanks", "rankBase", "dtype", "count", "sliceTiles", "slotBytes", "regionBOffset"):
                assert getattr(a, field) == getattr(alone, field), field
            assert bytes(a.codec) == bytes(cfg.to_c(xs[0].dtype)) and ranks == n
            assert a.epoch == 1 + turn and a.timeoutNs == int((5.0 + i) * 1e6)
            assert [a.inp[r] for r in range(n)] == [x.data_ptr() for x in xs] and [a.out[r] for r in range(n)] == [o.data_ptr() for o in outs]
            assert (a.trace[0] is not None) == (turn == 0 and i == 0)
            assert all(a.inp[r] is None for r in range(n, _lib.MAX_RANKS))


def test_a_codec_described_by_another_object_is_asked_each_time(recorder):
    class Described:
        group = 128

        def to_c(self, dtype):
            return C.CodecConfig("sdp4bit", 4, self.group).to_c(dtype)
    cfg, state = Described(), {}
    for group in (128, 32):
        cfg.group = group
        K.emulate_collective("reduce_scatter", _inputs(4), cfg, state=state)
        args, _ = recorder.launched[-1]
        assert args.codec.group == group and args.slotBytes == K.slot_bytes(cfg, 128, torch.float32)

"""A kernel layout that is still being written: what its first uses do (no GPU: stand-ins for the event and the kernels)."""
import copy
import pickle
import types

import pytest
import torch

from atlasinfer_b200.integration import atlas_wrappers as aw


class Ready:
    """Stands for the event behind a layout: the work it waits for is done after ``left`` more looks."""

    stream = 0, 7

    def __init__(self, left, log=None):
        self.left, self.log = left, log if log is not None else []

    def wait(self):
        self.left -= 1
        return self.left < 0

    def done(self):
        return self.left <= 0

    def finish(self):
        self.left = 0
        self.log.append("finish")


class Buffer(torch.Tensor):
    """A buffer of a layout that notes when it is copied or pickled."""

    log = []

    def __deepcopy__(self, memo):
        self.log.append("buffer")
        return self

    def __reduce_ex__(self, protocol):
        self.log.append("buffer")
        return super().__reduce_ex__(protocol)


def _layout(ready, n=128, k=64, source=None):
    tiles, scales = torch.zeros(n * k, dtype=torch.uint8), torch.zeros(n, dtype=torch.float16)
    none = torch.zeros(0, dtype=torch.int32)
    return aw.KernelLayout(source, tiles, scales, none, none, none, none.half(), n, k, 64, ready)


@pytest.fixture
def launches(monkeypatch):
    """(rows, launched plainly) of every linear that would have been launched."""
    seen = []

    def linear(x, *args):
        seen.append((x.shape[0], args[-1]))
        return x.new_zeros(x.shape[0], 128)

    monkeypatch.setattr(aw._capi, "native", lambda: types.SimpleNamespace(linear=linear))
    monkeypatch.setattr(aw, "status_word", lambda dev: None)
    return seen


@pytest.mark.parametrize("m", [1, 40, 300])
@pytest.mark.parametrize("left", [0, 1, 2])
def test_linears_are_launched_plainly_until_the_layout_is_final(m, left, launches):
    lay, x = _layout([Ready(left)]), torch.zeros(m, 64, dtype=torch.float16)
    for _ in range(4):
        aw.quantized_linear_forward(x, lay, None)
    assert launches == [(m, i < left) for i in range(4)]
    aw.quantized_linear_forward(x, _layout(None), None)
    assert launches[-1] == (m, False)


@pytest.mark.parametrize("left", [0, 1])
def test_streaming_form_is_launched_plainly_until_the_layout_is_final(left, monkeypatch):
    state, seen = [0], []
    lib = types.SimpleNamespace(
        atlas_qlinear_plain_launch=lambda on: state.append(on) or state[-2],
        atlas_qlinear_stream=lambda *a: seen.append(state[-1]) or 0)
    monkeypatch.setattr(aw._capi, "load", lambda: lib)
    monkeypatch.setattr(aw._capi, "stream_ptr", lambda dev: 0)
    monkeypatch.setattr(aw, "stream_workspace", lambda dev: torch.zeros(1))
    monkeypatch.setattr(aw, "status_word", lambda dev: torch.zeros(1))
    monkeypatch.setattr(aw.torch.cuda, "device", lambda dev: torch.no_grad())
    lay, x = _layout([Ready(left)]), torch.zeros(2, 64, dtype=torch.float16)
    for _ in range(3):
        aw.quantized_linear_forward(x, lay, None, force="stream")
    aw.quantized_linear_forward(x, lay, torch.zeros(128), force="stream")   # the conversion of the bias is in front
    assert seen == [int(i < left) for i in range(3)] + [1] and state[-1] == 0


@pytest.fixture
def events(monkeypatch):
    """The events of the layouts that ``_enqueued`` is asked for, on the stream that the list's last entry names."""
    made, on = [], [(0, 1)]

    def ready():
        made.append(Ready(1))
        made[-1].stream = on[-1]
        return made[-1]

    monkeypatch.setattr(aw._capi, "native", lambda: types.SimpleNamespace(LayoutReady=ready))
    monkeypatch.setattr(aw.torch.cuda, "device", lambda dev: torch.no_grad())
    monkeypatch.setattr(aw, "_cells", {})
    return made, on


def test_layouts_of_a_stream_become_final_together(events):
    made, on = events
    first = [_layout(aw._enqueued(None)) for _ in range(3)]
    on.append((0, 2))
    other = _layout(aw._enqueued(None))
    assert first[0].ready is first[1].ready is first[2].ready and first[0].ready == [made[2]]
    assert other.ready is not first[0].ready
    assert aw._pending(first[1]) and first[1].ready
    assert not aw._pending(first[1])                       # the second look finds the last event done
    assert not any(lay.ready for lay in first) and other.ready and aw._cells[0, 2] is other.ready
    on.append((0, 1))
    late = _layout(aw._enqueued(None))
    assert late.ready and not any(lay.ready for lay in first)   # what is final stays so


def test_a_layout_that_comes_during_the_look_is_not_taken_for_final(events):
    made, _ = events
    lay = _layout(aw._enqueued(None))
    made[0].left = 0
    later = []
    made[0].wait = lambda: later.append(_layout(aw._enqueued(None))) or True
    assert not aw._pending(lay)
    assert later[0].ready == [made[1]] and aw._pending(later[0])


def test_cells_of_streams_that_go_are_given_back(events):
    made, on = events
    lays = []
    for i in range(100):
        on.append((0, i))
        lays.append(_layout(aw._enqueued(None)))
        made[-1].left = 0 if i % 2 else 1
        if i % 2 == 0:
            aw._pending(lays[-1]), aw._pending(lays[-1])
    assert len(aw._cells) <= 16 and not lays[0].ready and not lays[1].ready and lays[-1].ready


def _copies(thing):
    """What ``thing()`` gives, copied and pickled, each with what happened in which order."""
    for make in (copy.deepcopy, lambda t: pickle.loads(pickle.dumps(t))):
        one = thing()
        Buffer.log.clear()
        yield make(one), list(Buffer.log)


def _watched(source, **kw):
    lay = _layout([Ready(9, Buffer.log)], source=source, **kw)
    return lay._replace(tiles=lay.tiles.as_subclass(Buffer), scales_tiled=lay.scales_tiled.as_subclass(Buffer))


def test_a_copied_layout_is_final_before_its_first_buffer_is_read():
    for again, log in _copies(lambda: _watched(None)):
        assert log[0] == "finish" and log.count("finish") == 1 and "buffer" in log
        assert type(again) is aw.KernelLayout and again.ready is None and (again.n_rows, again.n_cols) == (128, 64)
        assert torch.equal(again.tiles, torch.zeros(128 * 64, dtype=torch.uint8))
    for again, log in _copies(lambda: _watched(None)._replace(ready=None)):
        assert "finish" not in log and again.ready is None
    assert not _watched(None)._replace(ready=[]).finished().ready


def test_copied_modules_and_groups_keep_their_layouts():
    for again, log in _copies(_two_joined_modules):
        assert log[0] == "finish" and "buffer" in log
        for mod in again:
            assert mod._has_layout_for(mod.quantized_weights) and mod._kernel_layout.ready is None
            assert mod._group.layout.ready is None and mod._group.members[mod._group_index] is mod


def _two_joined_modules():
    q = aw.QuantizedTensor(torch.zeros(128 * 64, dtype=torch.int8), torch.zeros(0, dtype=torch.float16),
                           torch.zeros(0, dtype=torch.long), torch.ones(128, dtype=torch.float16), torch.Size([128, 64]), 64)
    mods = [aw.QuantizedLinear(q, None), aw.QuantizedLinear(q._replace(block_size=64), None)]
    group = aw.fuse_linears(mods)
    lay = _watched((q, mods[1].quantized_weights), n=256)
    group.layout, group.offsets = lay, [0, 128]
    for i, mod in enumerate(mods):
        mod._kernel_layout = aw.slice_layout(lay, 128 * i, 128, mod.quantized_weights)
    return mods


def test_a_gathered_linear_takes_a_final_layout():
    from atlasinfer_b200 import peer

    arena = types.SimpleNamespace(world=1, rank=0, bases=[0], state_ptr=0, carve=lambda n: 0, flags_ptr=lambda d: 0,
                                  local_tensor=lambda off, shape, dtype: None)
    log = []
    lin = peer.GatheredLinear(arena, _layout([Ready(9, log)]), 4, torch.float16)
    assert log == ["finish"] and lin.layout.ready is None

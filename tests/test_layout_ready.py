"""A kernel layout that is still being written: what its first uses do (no GPU: stand-ins for the event and the kernels)."""
import types

import pytest
import torch

from atlasinfer_b200.integration import atlas_wrappers as aw


class Ready:
    """Stands for the event behind a layout: the work it waits for is done after ``left`` more looks."""

    def __init__(self, left, log=None):
        self.left, self.log = left, log if log is not None else []

    def wait(self):
        self.left -= 1
        return self.left < 0


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
    lay, x = _layout(Ready(left)), torch.zeros(m, 64, dtype=torch.float16)
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
    lay, x = _layout(Ready(left)), torch.zeros(2, 64, dtype=torch.float16)
    for _ in range(3):
        aw.quantized_linear_forward(x, lay, None, force="stream")
    aw.quantized_linear_forward(x, lay, torch.zeros(128), force="stream")   # the conversion of the bias is in front
    assert seen == [int(i < left) for i in range(3)] + [1] and state[-1] == 0

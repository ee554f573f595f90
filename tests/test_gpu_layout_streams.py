"""Layouts on many streams: one look settles those of its own stream, none of another's."""
import pytest
import torch

from atlasinfer_b200 import _capi

pytestmark = pytest.mark.gpu


def _busy(dev):
    a = torch.randn(4096, 4096, device=dev)
    for _ in range(40):
        a = a @ a * 1e-4
    return a


def test_one_look_settles_the_layouts_of_its_stream(cuda_device):
    native = _capi.native()
    one, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(one):
        _busy(cuda_device)
        first, second = native.LayoutReady(), native.LayoutReady()
        assert not first.wait() and not second.wait()
    with torch.cuda.stream(other):
        free = native.LayoutReady()
        free.finish()
        assert free.wait()
        late = native.LayoutReady()
        other.synchronize()
        assert late.wait()
    with torch.cuda.stream(one):
        assert not first.wait()        # the other stream's end says nothing about this one
        one.synchronize()
        assert second.wait() and first.wait()
        _busy(cuda_device)
        third = native.LayoutReady()
        assert first.wait() and not third.wait()
    with torch.cuda.stream(other):
        assert third.wait()            # waits on the host
    assert one.query()


def test_streams_come_and_go(cuda_device):
    native = _capi.native()
    kept = []
    for i in range(100):
        with torch.cuda.stream(torch.cuda.Stream(priority=-(i % 2))):
            kept.append(native.LayoutReady())
        if i % 3:
            kept.pop(i % len(kept))
    for ready in kept:
        ready.finish()
        assert ready.wait()

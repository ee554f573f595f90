"""Several tensors in one quantizer launch: every tensor's streams are those of the oracle, whatever lies beside it."""
import pytest
import torch

import atlasinfer_b200 as ab
from atlasinfer_b200 import _capi
from oracle import atlas_oracle as O
from tests.util import bits, config_weights

pytestmark = pytest.mark.gpu


def _check(tensors, got, bs, thr):
    for i, (w, q) in enumerate(zip(tensors, got)):
        want = O.quantize(w.cpu(), block_size=bs, z_threshold=thr)
        for a, b in zip(q[:4], want[:4]):
            a = a.cpu()
            assert a.shape == b.shape and torch.equal(bits(a), bits(b)), f"tensor {i} of {len(tensors)}: {tuple(w.shape)}"


# sizes around a block, a warp's share of a tile (1024), a tile (8192) and a look-back step (256 tiles)
@pytest.mark.parametrize("bs", [32, 64, 96, 128, 256])
@pytest.mark.parametrize("sizes", [
    [1, 31, 32, 33, 127, 129, 255, 257, 1023, 1024, 1025, 8191, 8192, 8193, 16384, 24577],
    [8192] * 17 + [5],                                   # more tensors than a launch takes
    [300 * 8192 + 77, 3, 8192 * 2, 700001, 40000],       # a long one first: its tiles are looked back over, the next start anew
])
def test_streams_of_a_batch(bs, sizes, cuda_device):
    g = torch.Generator().manual_seed(bs)
    flat = config_weights(1, sum(sizes) + 8 * len(sizes), 7 + bs).view(-1)
    dev = flat.to(cuda_device)
    tensors, views, at = [], [], 0
    for n in sizes:
        off = at + int(torch.randint(0, 8, (1,), generator=g))   # any alignment of the input
        tensors.append(flat[off:off + n])
        views.append(dev[off:off + n])
        at += n + 8
    _check(tensors, ab.quantize_tensors(views, block_size=bs), bs, 3.0)


def test_blocks_with_subnormal_scales_beside_ordinary_ones(cuda_device):
    """The clamp of the codes is only applied where a warp's blocks need it: both forms in one tile."""
    w = config_weights(64, 256, 3)
    w[::3] *= 1e-4       # scales of a few fp16 subnormal steps
    w[1::7] = 0.0
    _check([w], ab.quantize_tensors([w.to(cuda_device)], block_size=128), 128, 3.0)


@pytest.mark.parametrize("bytes_", [0, 1, 2, 15, 16, 17, 4096, 70003])
@pytest.mark.parametrize("offset", [0, 2, 5])
def test_copy_many(bytes_, offset, cuda_device):
    L = _capi.load()
    src = torch.randint(0, 256, (40, 70100), dtype=torch.uint8, device=cuda_device)   # more copies than a launch takes
    dst = torch.full_like(src, 7)
    items = (_capi.CopyItem * 40)()
    for i, it in enumerate(items):
        it.dst, it.src, it.bytes = dst[i].data_ptr() + offset, src[i].data_ptr() + (offset if i % 2 else 0), bytes_
    _capi.check(L.atlas_copy_many(40, items, _capi.stream_ptr(cuda_device)), "atlas_copy_many")
    want = torch.full_like(src, 7)
    for i in range(40):
        s = offset if i % 2 else 0
        want[i, offset:offset + bytes_] = src[i, s:s + bytes_]
    assert torch.equal(dst, want)

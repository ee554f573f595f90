"""The dequantizer and the kernel layout at the edges of their 8192-element spans, byte for byte."""
import numpy as np
import pytest
import torch

import atlasinfer_b200 as ab
from atlasinfer_b200 import _capi
from atlasinfer_b200.integration import atlas_wrappers as aw
from atlasinfer_b200.quant import adaptive_quantizer as aq
from oracle import atlas_oracle as O
from tests.util import bits, config_weights

pytestmark = pytest.mark.gpu


def _streams(numel, bs, share, seed):
    """Streams of a padded tensor with ``share`` of its positions as outliers (any block size)."""
    gen = torch.Generator().manual_seed(seed)
    nb = -(-numel // bs)
    padded = nb * bs
    out = torch.rand(padded, generator=gen) < share
    idx = out.nonzero().flatten()
    codes = torch.randint(-127, 128, (padded - idx.numel(),), generator=gen).to(torch.int8)
    vals = torch.randn(idx.numel(), generator=gen).half()
    scales = (torch.rand(nb, generator=gen) * 1e-3 + 1e-6).half()
    return O.OracleQuantized(codes, vals, idx, scales, torch.Size([numel]), bs)


@pytest.mark.parametrize("numel", [1, 7, 8, 9, 8191, 8192, 8193, 16383, 16384, 16385, 16384 + 5, 32767, 32768, 32769, 100003])
@pytest.mark.parametrize("bs,share", [(128, 0.003), (64, 0.3), (100, 0.01), (7, 0.02), (32, 0.0), (32, 1.0)])
def test_dequantize_span_edges(numel, bs, share, cuda_device):
    o = _streams(numel, bs, share, numel + bs)
    got = aq._dequantize_on_device(ab.QuantizedTensor(*o).to(cuda_device), cuda_device)
    assert torch.equal(bits(got.cpu()), bits(O.dequantize(o)))


# blocks of whole units and others, whole spans and a last one that ends inside a unit, outputs on any boundary
@pytest.mark.parametrize("numel", [3 * 8192, 3 * 8192 + 20, 40000])
@pytest.mark.parametrize("bs", [4, 8, 24, 96, 100, 128, 160, 288, 20000])
@pytest.mark.parametrize("share", [0.003, 0.06])   # outliers searched for and marked
@pytest.mark.parametrize("off", [0, 1, 4, 8])
def test_dequantize_every_block_and_alignment(numel, bs, share, off, cuda_device):
    o = _streams(numel, bs, share, numel + bs)
    q, room = ab.QuantizedTensor(*o).to(cuda_device), torch.full((numel + 16,), 7, dtype=torch.float16, device=cuda_device)
    _capi.check(_capi.load().atlas_dequantize(
        _capi.ptr(q.fp8_data), q.fp8_data.numel(), _capi.ptr(q.fp16_outliers), _capi.ptr(q.outlier_indices), q.outlier_indices.numel(),
        q.scale_factors.data_ptr(), numel, bs, room.data_ptr() + 2 * off, _capi.stream_ptr(cuda_device)), "atlas_dequantize")
    room = room.cpu()
    assert torch.equal(bits(room[off:off + numel]), bits(O.dequantize(o)))
    assert (room[:off] == 7).all() and (room[off + numel:] == 7).all()


def _clustered(n, k, bs, clusters, seed):
    """Streams of an [n, k] tensor whose outliers fill ``clusters`` (first position, length, every how many)."""
    gen = torch.Generator().manual_seed(seed)
    out = torch.zeros(n * k, dtype=torch.bool)
    for first, length, step in clusters:
        out[first:first + length:step] = True
    idx = out.nonzero().flatten()
    codes = torch.randint(-127, 128, (n * k - idx.numel(),), generator=gen).to(torch.int8)
    scales = (torch.rand(n * k // bs, generator=gen) * 1e-3 + 1e-6).half()
    return O.OracleQuantized(codes, torch.randn(idx.numel(), generator=gen).half(), idx, scales, torch.Size([n, k]), bs)


# long runs of spans without outliers before, between and behind clusters of more of them than are searched for
@pytest.mark.parametrize("clusters", [
    [(0, 2000, 1)], [(300 * 4096 - 2000, 2000, 1)], [(40 * 8192 - 1, 4000, 2), (120 * 8192 + 8191, 2, 1)],
    [(17, 1, 1), (50 * 8192, 8192, 1), (58 * 8192, 8192, 3), (100 * 8192 + 5, 1, 1)], [(i * 32 * 8192 - 64, 700, 3) for i in range(1, 5)]])
@pytest.mark.parametrize("bs", [128, 64])
def test_clusters_of_outliers(clusters, bs, cuda_device):
    o = _clustered(300, 4096, bs, clusters, bs)
    assert o.outlier_indices.numel() > 900
    q = ab.QuantizedTensor(*o).to(cuda_device)
    assert torch.equal(bits(aq._dequantize_on_device(q, cuda_device).cpu()), bits(O.dequantize(o)))
    _assert_layout(aw.build_kernel_layout(q), _layout_reference(o))


@pytest.mark.parametrize("damage", ["shuffled", "reversed", "negative", "beyond", "equal"])
def test_damaged_indices_stay_inside_the_output(damage, cuda_device):
    """The values are arbitrary, but nothing outside the buffers is written, and a layout points into its own lists."""
    o = _clustered(300, 4096, 128, [(100 * 8192, 3000, 1)], 9)
    idx = o.outlier_indices.clone()
    if damage == "shuffled":
        idx = idx[torch.randperm(idx.numel(), generator=torch.Generator().manual_seed(2))]
    elif damage == "reversed":
        idx = idx.flip(0)
    elif damage == "negative":
        idx[1500] = -(1 << 40)
    elif damage == "beyond":
        idx[1500:] = 1 << 60
    else:
        idx[:] = idx[0]
    q, numel = ab.QuantizedTensor(*o._replace(outlier_indices=idx)).to(cuda_device), 300 * 4096
    room = torch.full((numel + 4096,), 7, dtype=torch.float16, device=cuda_device)
    _capi.check(_capi.load().atlas_dequantize(
        q.fp8_data.data_ptr(), q.fp8_data.numel(), q.fp16_outliers.data_ptr(), q.outlier_indices.data_ptr(), idx.numel(),
        q.scale_factors.data_ptr(), numel, 128, room.data_ptr() + 4096, _capi.stream_ptr(cuda_device)), "atlas_dequantize")
    assert (room[:2048] == 7).all() and (room[2048 + numel:] == 7).all()
    lay = aw.build_kernel_layout(q)
    again = aw.build_kernel_layout(q)
    assert torch.equal(lay.chunk_ptr, again.chunk_ptr)
    assert int(lay.chunk_ptr.min()) >= 0 and int(lay.chunk_ptr.max()) <= idx.numel()


@pytest.mark.parametrize("off", [1, 5, 15])
def test_dequantize_unaligned_codes(off, cuda_device):
    o = _streams(30000, 128, 0.01, off)
    room = torch.zeros(off + o.fp8_data.numel(), dtype=torch.int8, device=cuda_device)
    room[off:] = o.fp8_data.to(cuda_device)
    q = ab.QuantizedTensor(*o).to(cuda_device)._replace(fp8_data=room[off:])
    got = aq._dequantize_on_device(q, cuda_device)
    assert torch.equal(bits(got.cpu()), bits(O.dequantize(o)))


def _layout_reference(o):
    """What the layout holds, from the streams: tiles, scales, row_ptr, chunk_ptr, entries, values."""
    (n, k), bs = o.original_shape, o.block_size
    n_pad = -(-n // 128) * 128
    dense = np.full(n_pad * k, 128, np.uint8)
    idx, codes = o.outlier_indices.numpy(), o.fp8_data.numpy()
    keep = np.ones(n * k, bool)
    keep[idx] = False
    dense[:n * k][keep] = (codes.astype(np.int16) + 128).astype(np.uint8)
    tiles = dense.reshape(n_pad // 128, 128, k // 64, 64).transpose(0, 2, 1, 3)
    scales = np.zeros((n_pad, k // bs), np.int16)
    scales[:n] = o.scale_factors.view(torch.int16).numpy().reshape(n, k // bs)
    scales = scales.reshape(n_pad // 128, 128, k // bs).transpose(0, 2, 1)
    row, col = idx // k, idx % k
    row_ptr = np.searchsorted(idx, np.arange(n + 1) * k)
    order = np.lexsort((row, col, row // 16))
    entries = ((row % 16) << 24 | col)[order]
    strip = (row // 16)[order]
    key = strip * (k + 1) + col[order]
    chunk_ptr = np.searchsorted(key, (np.arange(n_pad // 16)[:, None] * (k + 1) + np.arange(k // 64 + 1) * 64).ravel())
    return tiles.ravel(), scales.ravel(), row_ptr, chunk_ptr, entries, o.fp16_outliers.view(torch.int16).numpy()[order]


def _assert_layout(lay, want, row_ptr=True):
    got = [lay.tiles, lay.scales_tiled.view(torch.int16), lay.row_ptr, lay.chunk_ptr, lay.entries, lay.vals_sorted.view(torch.int16)]
    for name, g, w in zip(("tiles", "scales", "row_ptr", "chunk_ptr", "entries", "values"), got, want):
        if name != "row_ptr" or row_ptr:
            assert np.array_equal(g.cpu().numpy().astype(np.int64), np.asarray(w).astype(np.int64)), name


# one-unit rows, rows and columns on neither 16 nor 128, more than RP_STRIP_CAP outliers in a strip, many scale blocks,
# one and two whole spans, a span and one row more
@pytest.mark.parametrize("n,k,bs,thr", [(1, 64, 64, 3.0), (16, 64, 16, 3.0), (129, 192, 64, 3.0), (300, 1088, 32, 3.0),
                                        (200, 4096, 128, 1.0), (128, 8192, 128, 0.5), (77, 11008, 256, 3.0),
                                        (4, 4096, 128, 3.0), (8, 4096, 64, 1.0), (257, 64, 64, 3.0), (1, 16448, 64, 1.0)])
def test_repack_matches_streams(n, k, bs, thr, cuda_device):
    w = config_weights(n, k, n + k)
    o = O.quantize(w, max(bs, 32), thr)._replace() if bs >= 32 else _streams(n * k, bs, 0.01, 3)._replace(original_shape=torch.Size([n, k]))
    lay = aw.build_kernel_layout(ab.QuantizedTensor(*o).to(cuda_device))
    _assert_layout(lay, _layout_reference(o))


@pytest.mark.parametrize("count", [2, 9])   # 9: more than one launch takes
def test_joined_layout_equals_concatenated(count, cuda_device):
    qs = [ab.QuantizedTensor(*O.quantize(config_weights(n, 512, n), 128, 3.0)).to(cuda_device)
          for n in (100, 256, 16, 130, 1, 384, 127, 129, 64)[:count]]
    joined, offsets = aw.build_joined_layout(qs)
    parts = [aw.build_kernel_layout(q) for q in qs]
    whole = aw.concat_layouts(parts)
    assert offsets == [sum(p.tiles.numel() // 512 for p in parts[:i]) for i in range(count)]
    assert (joined.n_rows, joined.n_cols, joined.block_size) == (whole.n_rows, whole.n_cols, whole.block_size)
    for f in ("tiles", "scales_tiled", "chunk_ptr", "entries", "vals_sorted"):
        assert torch.equal(bits(getattr(joined, f)), bits(getattr(whole, f))), f

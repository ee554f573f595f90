"""The linear kernels at the edges of their token tiles, K slices and strip pairs.

Outputs are held to max|err| <= 1e-2 * rms(ref) like the other linear tests (tests/util.py).
"""
import pytest
import torch

import atlasinfer_b200 as ab
from atlasinfer_b200.integration import atlas_wrappers as aw
from oracle import atlas_oracle as O
from tests.util import config_weights, rel_max_err

pytestmark = pytest.mark.gpu
LINEAR_TOL = 1e-2


def _check(n, k, ms, dev, bs=128, thr=3.0, force=None, strided=False):
    o = O.quantize(config_weights(n, k, n + k), bs, thr)
    lay = aw.build_kernel_layout(ab.QuantizedTensor(*o).to(dev))
    w = O.dequantize(o)
    gen = torch.Generator().manual_seed(n)
    b = (torch.randn(n, generator=gen) * 0.02).half()
    for m in ms:
        for dtype in (torch.float16, torch.bfloat16):
            x = torch.randn(m, k + (1 if strided else 0), generator=gen).to(dtype)
            xd = x.to(dev)[:, :k]      # rows on no 16-byte boundary when strided
            y = aw.quantized_linear_forward(xd, lay, b.to(dev), force)
            aw.check_status(dev)
            err = rel_max_err(y, O.linear(x[:, :k].contiguous(), w, b), report=f"{n}x{k} bs={bs} m={m}")
            assert err < LINEAR_TOL, f"{n}x{k} bs={bs} m={m} {dtype}: {err}"


# one row of one tile, ragged rows, one k-tile (a phase of the dequantizers without work), K slices of unequal length,
# blocks smaller than, not commensurable with and larger than a k-tile
@pytest.mark.parametrize("n,k,bs", [(1, 64, 64), (16, 64, 32), (129, 192, 64), (200, 1088, 32), (500, 1024, 256),
                                    (300, 576, 96), (128, 4096, 128), (1100, 2112, 64)])
def test_tile_kernel_edges(n, k, bs, cuda_device):
    _check(n, k, (1, 16, 17, 32, 33, 64, 65, 96, 97, 128), cuda_device, bs=bs, force="gemm")


@pytest.mark.parametrize("thr", [0.5, 1.0, 1.5])
def test_tile_kernel_dense_outliers(thr, cuda_device):
    _check(256, 1024, (17, 33, 96, 128), cuda_device, thr=thr, force="gemm")   # more than 16 per strip and k-tile


def test_tile_kernel_unaligned_rows(cuda_device):
    _check(200, 512, (17, 64, 100), cuda_device, strided=True)


# up to 128 rows that the prompt kernel takes: a long K under few row tiles (16 K slices; an odd number of k-tiles, ragged
# rows, blocks smaller than and not commensurable with a k-tile), and one wave of 128-token tiles
@pytest.mark.parametrize("n,k,bs,thr,ms", [(1024, 8192, 128, 3.0, (17, 33, 64)), (130, 16448, 64, 3.0, (17, 32, 40)),
                                           (512, 12288, 96, 3.0, (32, 64)), (256, 16384, 32, 1.0, (20, 50)),
                                           (12288, 1088, 64, 3.0, (65, 128)), (9464, 1024, 32, 1.5, (97,))])
def test_prompt_kernel_takes_over(n, k, bs, thr, ms, cuda_device):
    _check(n, k, ms, cuda_device, bs=bs, thr=thr)
    if n <= 130:
        _check(n, k, ms[:1], cuda_device, bs=bs, thr=thr, strided=True)


# the same kernel with the gather of its output, one rank: one to many K slices, ragged rows, more than 16 outliers of a
# strip in a stage, every block form
@pytest.mark.parametrize("n,k,bs,thr", [(200, 8256, 64, 3.0), (1000, 2048, 32, 3.0), (128, 6144, 96, 1.0), (64, 64, 64, 3.0)])
def test_gathered_gemm_edges(n, k, bs, thr, cuda_device):
    from atlasinfer_b200 import peer
    o = O.quantize(config_weights(n, k, n + k), bs, thr)
    lay = aw.build_kernel_layout(ab.QuantizedTensor(*o).to(cuda_device))
    w = O.dequantize(o)
    gen = torch.Generator().manual_seed(n)
    b = (torch.randn(n, generator=gen) * 0.02).half()
    arena = peer.PeerArena(1 << 20, cuda_device, world=1, rank=0, exchange=False)
    try:
        for dtype in (torch.float16, torch.bfloat16):
            g = peer.GatheredLinear(arena, lay, 64, dtype, bias=b.to(cuda_device), kernel="gemm")
            for m in (1, 32, 33, 64):
                x = torch.randn(m, k, generator=gen).to(dtype)
                y = g(x.to(cuda_device), wait=True).clone()
                aw.check_status(cuda_device)
                err = rel_max_err(y, O.linear(x, w, b), report=f"gathered {n}x{k} bs={bs} m={m}")
                assert err < LINEAR_TOL, f"{n}x{k} bs={bs} m={m} {dtype}: {err}"
    finally:
        arena.close()


# prompts whose few row tiles are cut along K: second kernel, 8 features at a time or one
@pytest.mark.parametrize("n,k", [(128, 4096), (257, 2048), (1024, 8192)])
def test_prompt_k_slices(n, k, cuda_device):
    _check(n, k, (129, 256, 257, 301), cuda_device)


def test_back_to_back_launches(cuda_device):
    # consecutive launches overlap (programmatic dependent launch): many in a row, no synchronisation between them
    shapes = [(6144, 2048), (2048, 2048), (8192, 2048), (2048, 8192)]
    work = []
    for n, k in shapes:
        q = ab.quantize_tensor(config_weights(n, k, n).to(cuda_device))
        x = torch.randn(128, k, device=cuda_device).half()
        lay = aw.build_kernel_layout(q)
        work.append((lay, x, {m: aw.quantized_linear_forward(x[:m], lay, None) for m in (1, 20, 40, 96, 128)}))
        torch.cuda.synchronize()
    got = []
    for _ in range(20):
        for lay, x, want in work:
            for m in want:
                got.append((aw.quantized_linear_forward(x[:m], lay, None), want[m]))
    assert all(torch.equal(a, b) for a, b in got)
    aw.check_status(cuda_device)


# strips in pairs (the pairs fill the SMs, 12 chunks of K or more): an odd number of strips, ragged rows; and single ones
@pytest.mark.parametrize("n,k,bs", [(9441, 4096, 64), (9460, 3072, 128), (9441, 4352, 256), (9473, 256, 128)])
def test_strip_pairs(n, k, bs, cuda_device):
    _check(n, k, (1, 2, 3, 8), cuda_device, bs=bs, force="gemv")
    _check(n, k, (1,), cuda_device, bs=bs, thr=1.0, force="gemv")

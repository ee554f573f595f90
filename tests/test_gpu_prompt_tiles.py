"""Prompts of every token tile: one or two accumulators per rebuilt weight tile, tokens at the tiles' edges, odd k-tile counts
(rings that end inside a round), ragged feature counts, K slices."""
import ctypes

import pytest
import torch

import atlasinfer_b200 as ab
from atlasinfer_b200 import _capi
from atlasinfer_b200.integration import atlas_wrappers as aw
from tests.test_prompt_plan import RUNS
from tests.util import config_weights

pytestmark = pytest.mark.gpu

_layouts = {}


def _weight(n, k, dev):
    if (n, k) not in _layouts:
        _layouts.clear()
        q = ab.quantize_tensor(config_weights(n, k, n + k).to(dev))
        w = ab.dequantize_tensor(q, dev).double()
        ab.clear_dequantized_cache()
        _layouts[n, k] = aw.build_kernel_layout(q), w
    return _layouts[n, k]


@pytest.mark.parametrize("m", [129, 160, 161, 192, 224, 225, 257, 300, 320, 321, 384, 385, 500, 769, 1152])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n,k", [(11008, 1024), (11000, 2176), (1100, 4224), (6144, 640), (20000, 512), (2048, 8192)])
def test_prompt_matches_fp64(n, k, m, dtype, cuda_device):
    lay, w = _weight(n, k, cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(m)
    x = torch.randn(m, k, generator=g, device=cuda_device).to(dtype)
    bias = (torch.randn(n, generator=g, device=cuda_device) * 0.02).half()
    y = aw.quantized_linear_forward(x, lay, bias).double()
    r = x.double() @ w.t() + bias.double()
    # the rounding of the output type: half a unit in its last place, and fp32 sums of K products of 2^-24 each beside it
    ulp = 2.0 ** -11 if dtype is torch.float16 else 2.0 ** -8
    rms = r.pow(2).mean().sqrt()
    assert ((y - r).abs() <= ulp * r.abs() + 1e-3 * rms).all()
    aw.check_status(cuda_device)


@pytest.mark.parametrize("tokens,m,n,k", [(t, *run) for t in sorted(RUNS) for run in RUNS[t]])
def test_every_tile_at_every_place_of_its_rings(tokens, m, n, k, cuda_device):
    chosen, slices = ctypes.c_int(), ctypes.c_int()
    _capi.check(_capi.load().atlas_qlinear_gemm_plan(m, n, k, ctypes.byref(chosen), ctypes.byref(slices)), "atlas_qlinear_gemm_plan")
    assert chosen.value == tokens
    g = torch.Generator(device=cuda_device).manual_seed(n + k)
    w = torch.randn(n, k, generator=g, device=cuda_device) * 0.02
    w.view(-1)[::1009] = 0.4   # outliers of the blocks they are in
    q = ab.quantize_tensor(w.half(), block_size=64)
    x = torch.randn(m, k, generator=g, device=cuda_device).half()
    y = aw.quantized_linear_forward(x, aw.build_kernel_layout(q), None).double()
    r = x.double() @ ab.dequantize_tensor(q, cuda_device).double().t()
    ab.clear_dequantized_cache()
    # half a unit of the output type in its last place, and fp32 sums of K products of 2^-24 each beside it
    assert ((y - r).abs() <= 2.0 ** -11 * r.abs() + 1e-3 * r.pow(2).mean().sqrt()).all()
    aw.check_status(cuda_device)

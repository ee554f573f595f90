"""A module's kernel layout is used while it may still be written: on its own stream, on another, in a capture, in a copy."""
import copy
import pickle

import pytest
import torch

import atlasinfer_b200 as ab
from tests.util import config_weights

pytestmark = pytest.mark.gpu


def _modules(dev, fused, seed=5):
    g = torch.Generator().manual_seed(seed)
    ws = [config_weights(n, 1024, seed + i).to(dev) for i, n in enumerate((512, 200, 1300))]
    mods = [ab.QuantizedLinear(q, (torch.randn(w.shape[0], generator=g) * 0.02).half().to(dev)) for q, w in zip(ab.quantize_tensors(ws), ws)]
    if fused:
        ab.fuse_linears(mods)
    return mods


def _want(mods, x):
    out = []
    for m in mods:
        w = ab.dequantize_tensor(m.quantized_weights, x.device).double()
        out.append(x.double() @ w.t() + m.bias.double())
    ab.clear_dequantized_cache()
    return out


def _check(got, want):
    for y, r in zip(got, want):
        assert (y.double() - r).abs().max().item() < 1e-2 * r.pow(2).mean().sqrt().item()


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("m", [1, 40, 300])
@pytest.mark.parametrize("how", ["same", "other", "capture", "copied", "pickled", "copied elsewhere", "pickled elsewhere", "freed"])
def test_first_uses_of_a_layout(fused, m, how, cuda_device):
    x = torch.randn(m, 1024, device=cuda_device).half()
    mods = _modules(cuda_device, fused)
    want = _want(mods, x)
    torch.cuda.synchronize()
    busy = torch.randn(4096, 4096, device=cuda_device)
    with torch.no_grad():
        for _ in range(20):
            busy = busy @ busy * 1e-4      # the stream has work in front of the layouts
        first = [mod(x) for mod in mods]   # enqueues them
        if how == "same":
            got = [mod(x) for mod in mods]
        elif how == "other":
            side = torch.cuda.Stream()
            with torch.cuda.stream(side):
                got = [mod(x) for mod in mods]
            side.synchronize()
        elif how == "capture":
            graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
            with torch.cuda.stream(side):
                graph.capture_begin()
                got = [mod(x) for mod in mods]
                graph.capture_end()
            graph.replay()
        elif how == "freed":
            for mod in mods:
                mod.offload_canonical()
            trash = [torch.full((1 << 20,), 77, dtype=torch.int8, device=cuda_device) for _ in range(16)]
            got = [mod(x) for mod in mods]
            del trash
        else:
            # (on a stream that nothing orders behind the one that writes the layouts)
            side = torch.cuda.Stream() if how.endswith("elsewhere") else torch.cuda.current_stream()
            with torch.cuda.stream(side):
                again = copy.deepcopy(mods) if how.startswith("copied") else pickle.loads(pickle.dumps(mods))
                got = [mod(x) for mod in again]
            side.synchronize()
    torch.cuda.synchronize()
    _check(first, want)
    _check(got, want)

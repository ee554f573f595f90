"""What may start under the kernel in front of it: a captured graph tells an ordinary launch from a programmatic one."""
import ctypes

import pytest
import torch

import atlasinfer_b200 as ab
from atlasinfer_b200 import _capi
from atlasinfer_b200.integration import atlas_wrappers as aw
from tests.util import bits, config_weights

pytestmark = pytest.mark.gpu


def _edges(dev, front, fn):
    """Of a capture of ``fn`` behind ``front``: how many kernels wait for the end of the one in front of them, and how many
    may start before it."""
    graph, side = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream(dev)
    with torch.cuda.stream(side):
        graph.capture_begin()
        front()
        fn()
        graph.capture_end()
    cuda, handle, count = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(64)
    nodes, data = (ctypes.c_void_p * 64)(), (ctypes.c_ubyte * 8 * 64)()   # CUgraphEdgeData: two ports, the type, padding
    assert cuda.cuGraphGetEdges_v2(handle, nodes, (ctypes.c_void_p * 64)(), data, ctypes.byref(count)) == 0
    early = sum(data[i][2] == 1 for i in range(count.value))   # CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC
    return count.value - early, early


# the per-strip kernel in one and in two tiles, the streaming kernel, the tile kernel, the prompt kernel with its copy
@pytest.mark.parametrize("m,force", [(1, None), (16, None), (4, "stream"), (40, None), (100, None), (300, None)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_every_kernel_of_a_linear_can_be_launched_plainly(m, force, dtype, cuda_device):
    L = _capi.load()
    lay = aw.build_kernel_layout(ab.quantize_tensor(config_weights(1024, 2048, 9).to(cuda_device)))
    x = torch.randn(m, 2048, device=cuda_device).to(dtype)
    want = aw.quantized_linear_forward(x, lay, None, force)
    torch.cuda.synchronize()
    def linear():
        aw.quantized_linear_forward(x, lay, None, force)

    def plain():
        assert L.atlas_qlinear_plain_launch(1) == 0
        linear()
        assert L.atlas_qlinear_plain_launch(0) == 1

    ordinary, early = _edges(cuda_device, linear, linear)   # kernels of both calls but the first
    assert ordinary == 0 and early % 2 == 1
    kernels = (early + 1) // 2
    assert _edges(cuda_device, linear, plain) == (kernels, kernels - 1)
    L.atlas_qlinear_plain_launch(1)
    got = aw.quantized_linear_forward(x, lay, None, force)
    L.atlas_qlinear_plain_launch(0)
    assert torch.equal(bits(got), bits(want))


@pytest.mark.parametrize("m,force", [(1, None), (4, "stream"), (40, None), (300, None)])
def test_a_bias_converted_in_the_call_is_waited_for(m, force, cuda_device):
    lay = aw.build_kernel_layout(ab.quantize_tensor(config_weights(1024, 2048, 9).to(cuda_device)))
    x, bias = torch.randn(m, 2048, device=cuda_device).half(), torch.randn(1024, device=cuda_device)
    want = aw.quantized_linear_forward(x, lay, bias.half(), force)
    assert torch.equal(bits(aw.quantized_linear_forward(x, lay, bias, force)), bits(want))
    assert _edges(cuda_device, lambda: torch.cuda._sleep(1), lambda: aw.quantized_linear_forward(x, lay, bias, force))[1] == 0

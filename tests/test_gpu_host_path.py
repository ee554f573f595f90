"""The native host path on other streams and threads than the default, and the quantizer's second attempt."""
import threading

import pytest
import torch

import atlasinfer_b200 as ab
from atlasinfer_b200.integration import atlas_wrappers as aw
from oracle import atlas_oracle as O
from tests.util import assert_streams_equal, bits, config_weights

pytestmark = pytest.mark.gpu


def _slow_copy(t, dev):
    """``t`` on ``dev``, written by the current stream behind a few milliseconds of other work."""
    a = torch.ones(4096, 4096, device=dev)
    for _ in range(20):
        a = a @ a * 0.0
    return t.to(dev) + a[0, 0].to(t.dtype)


# rows of the per-strip kernel, of the tile kernel, of the prompt kernel with its workspace
@pytest.mark.parametrize("m", [1, 40, 160])
def test_linear_follows_the_current_stream(m, cuda_device):
    layer = ab.QuantizedLinear(ab.quantize_tensor(config_weights(512, 1024, 1).to(cuda_device)),
                               torch.linspace(-1, 1, 512, device=cuda_device).half())
    x = torch.randn(m, 1024, generator=torch.Generator().manual_seed(m)).to(torch.bfloat16)
    want = layer(x.to(cuda_device))
    torch.cuda.synchronize()
    side = torch.cuda.Stream(cuda_device)
    with torch.cuda.stream(side):
        y = layer(_slow_copy(x, cuda_device))
        y.record_stream(side)
    side.synchronize()
    assert torch.equal(bits(y), bits(want))


def test_quantizer_follows_the_current_stream(cuda_device):
    ws = [config_weights(300, 256, 2), config_weights(64, 1024, 3)]
    side = torch.cuda.Stream(cuda_device)
    with torch.cuda.stream(side):
        qs = ab.quantize_tensors([_slow_copy(w, cuda_device) for w in ws])
    side.synchronize()
    for q, w in zip(qs, ws):
        assert_streams_equal(q, O.quantize(w))


def test_threads_do_not_disturb_each_other(cuda_device):
    jobs, errors = [], []
    for i, (n, k) in enumerate([(512, 1024), (2048, 512), (256, 4096), (1024, 2048)]):
        w = config_weights(n, k, i)
        o = O.quantize(w)
        lay = aw.build_kernel_layout(ab.QuantizedTensor(*o).to(cuda_device))
        xs = [torch.randn(m, k, device=cuda_device).half() for m in (1, 24, 100, 300)]
        jobs.append((w.to(cuda_device), o, lay, xs, [aw.quantized_linear_forward(x, lay, None) for x in xs]))
    torch.cuda.synchronize()

    def work(job):
        try:
            w, o, lay, xs, want = job
            stream = torch.cuda.Stream(cuda_device)
            with torch.cuda.stream(stream):
                for _ in range(10):
                    q = ab.quantize_tensor(w)
                    ys = [aw.quantized_linear_forward(x, lay, None) for x in xs]
                    stream.synchronize()
                    assert_streams_equal(q, o)
                    assert all(torch.equal(bits(a), bits(b)) for a, b in zip(ys, want))
        except BaseException as e:   # noqa: BLE001 - reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(job,)) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    aw.check_status(cuda_device)


def test_one_tensor_of_a_batch_overflows_its_outlier_buffer(cuda_device):
    # twelve entries of every 128 at +-1 among small ones: 9.4 % outliers, where the first buffer holds 3.1 % and 1024
    gen = torch.Generator().manual_seed(4)
    dense = torch.randn(1024, 128, generator=gen) * 1e-3
    dense[:, ::11] = torch.where(torch.rand(1024, 12, generator=gen) < 0.5, -1.0, 1.0)
    ws = [config_weights(64, 512, 5), dense.half(), config_weights(33, 257, 6)]
    qs = ab.quantize_tensors([w.to(cuda_device) for w in ws])
    assert qs[1].fp16_outliers.numel() > dense.numel() // 32 + 1024
    for q, w in zip(qs, ws):
        assert_streams_equal(q, O.quantize(w))


@pytest.mark.parametrize("m", [1, 24, 100, 160])
def test_first_call_of_a_thread_may_be_captured(m, cuda_device):
    # what a thread looks up once per device (attributes, occupancy, the kernels' choice) must not need a call before
    # the capture; the layout and the kernels' code are there already, as in a program that captures its second pass
    lay = aw.build_kernel_layout(ab.quantize_tensor(config_weights(1024, 2048, 9).to(cuda_device)))
    x = torch.randn(m, 2048, device=cuda_device).to(torch.bfloat16)
    want = aw.quantized_linear_forward(x, lay, None)
    torch.cuda.synchronize()
    got, errors = [], []

    def work():
        try:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.stream(torch.cuda.Stream(cuda_device)):
                with torch.cuda.graph(graph):
                    y = aw.quantized_linear_forward(x, lay, None)
                graph.replay()
                torch.cuda.current_stream().synchronize()
            got.append(y.clone())
            torch.cuda.synchronize()
        except BaseException as e:   # noqa: BLE001 - reported by the main thread
            errors.append(e)

    thread = threading.Thread(target=work)
    thread.start()
    thread.join()
    assert not errors, errors[0]
    assert torch.equal(bits(got[0]), bits(want))

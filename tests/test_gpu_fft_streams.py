"""The first FP32 transform of a size where its tables must be in place before
they are read: on a non-blocking stream, from several threads on streams of their
own, and while a stream is captured.  Sizes that no other test has used, against
torch's FP64 transform (the bound of tests/test_gpu_fft_sizes.py)."""
import threading

import pytest

from tests.test_gpu_fft_sizes import TOL, _shifted

pytestmark = pytest.mark.gpu


def _image(n):
    import torch

    x = torch.randn(n, n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    return x, torch.zeros(n, n, dtype=torch.complex64, device="cuda")


def _to_grid(x, g, stream):
    from rc_gb300 import lib

    lib.check(lib.load().gb_image_to_grid_f32(x.data_ptr(), None, x.shape[0], g.data_ptr(),
                                              stream.cuda_stream), "gb_image_to_grid_f32")


def _check(x, g):
    import torch

    exp = _shifted(torch.fft.fft2, x.double())
    assert float(torch.linalg.norm(g - exp) / torch.linalg.norm(exp)) < TOL


@pytest.mark.parametrize("n", [48, 4032, 8064])
def test_first_use_on_a_side_stream(n):
    import torch

    x, g = _image(n)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    _to_grid(x, g, s)
    s.synchronize()
    _check(x, g)


def test_first_use_from_several_threads():
    import torch

    n, errors = 3840, []
    work = [_image(n) + (torch.cuda.Stream(),) for _ in range(6)]
    torch.cuda.synchronize()
    gate = threading.Barrier(len(work))

    def one(x, g, s):
        try:
            gate.wait()
            _to_grid(x, g, s)
            s.synchronize()
        except Exception as e:  # shown below
            errors.append(e)

    threads = [threading.Thread(target=one, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for x, g, _ in work:
        _check(x, g)


def test_first_use_while_its_stream_is_captured():
    import torch

    x, g = _image(1120)
    torch.cuda.synchronize()
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        _to_grid(x, g, s)
    assert float(g.abs().sum()) == 0.0  # captured, not run
    graph.replay()
    torch.cuda.synchronize()
    _check(x, g)

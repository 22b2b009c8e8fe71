"""Convolution layers called from several host threads, each on a stream of its own: the
calls of a device share one scratch, and each must give what it gives alone, bit for bit.
The grids differ, so that the scratch grows while other calls are under way."""
import ctypes as C
import threading

import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(9, 17, 21), (5, 40, 33), (17, 33, 33), (3, 50, 60)]


def _inputs(torch, k):
    V = SHAPES[k][0] * SHAPES[k][1] * SHAPES[k][2]
    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn(V, 16, generator=g, device="cuda").bfloat16()
    w = (0.1 * torch.randn(16, 16, 27, generator=g, device="cuda")).bfloat16()
    b = torch.randn(16, generator=g, device="cuda")
    gy = torch.randn(V, 16, generator=g, device="cuda")
    return x, w, b, gy


def _layer(torch, lib, k, inputs, stream):
    x, w, b, gy = inputs
    out = [torch.zeros_like(x), torch.zeros_like(gy), torch.zeros(16, 16, 27, device="cuda"), torch.zeros(16, device="cuda")]
    torch.cuda.current_stream().synchronize()
    p = lambda t: C.c_void_p(t.data_ptr())
    st = C.c_void_p(stream)
    assert lib.hrn_cnn_conv3d_forward(16, 16, *SHAPES[k], p(x), p(w), p(b), 1, p(out[0]), st) == 0
    assert lib.hrn_cnn_conv3d_backward(16, 16, *SHAPES[k], p(x), p(w), p(out[0]), 1, p(gy), p(out[1]), p(out[2]), p(out[3]), st) == 0
    return out


def test_layers_of_several_threads(gpu_lib):
    import torch
    inputs = [_inputs(torch, k) for k in range(len(SHAPES))]
    torch.cuda.synchronize()
    got = [[] for _ in SHAPES]
    errors = []

    def work(k):
        try:
            torch.cuda.set_device(0)
            with torch.cuda.stream(torch.cuda.Stream()) as _:
                st = torch.cuda.current_stream().cuda_stream
                for _ in range(20):
                    got[k].append(_layer(torch, gpu_lib, k, inputs[k], st))
        except BaseException as e:   # noqa: BLE001 -- shown by the assertion below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(SHAPES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    torch.cuda.synchronize()
    for k in range(len(SHAPES)):
        alone = _layer(torch, gpu_lib, k, inputs[k], torch.cuda.current_stream().cuda_stream)
        for out in got[k]:
            assert all(torch.equal(a, b) for a, b in zip(out, alone)), k

"""A scalar reduction asked for while its stream is under capture is refused, as every call
that synchronizes is, and the calls after it are not affected."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_first_reduction_under_capture(gpu_lib):
    import torch
    from hirensi_b200.solver import Solver
    rng = np.random.default_rng(1)
    h = rng.standard_normal(100000)
    x = torch.from_numpy(h).cuda()
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    out = C.c_double()
    p = C.c_void_p(x.data_ptr())
    rt = C.CDLL("libcudart.so.12")   # torch's, already loaded
    handle, graph = C.c_void_p(st.cuda_stream), C.c_void_p()
    # freed blocks of the workspace's size with other contents: what it may be cut from
    blocks = [C.c_void_p() for _ in range(2048)]
    for b in blocks:
        assert rt.cudaMalloc(C.byref(b), C.c_size_t(297 * 8)) == 0 and rt.cudaMemset(b, 7, C.c_size_t(297 * 8)) == 0
    torch.cuda.synchronize()
    for b in blocks[::2]:
        assert rt.cudaFree(b) == 0
    with Solver("fp64") as s:
        s.set_stream(st.cuda_stream)
        assert rt.cudaStreamBeginCapture(handle, 2) == 0   # relaxed: allocations are allowed
        rc = gpu_lib.hrn_vec_dot(s.h, x.numel(), p, p, C.byref(out))
        rt.cudaStreamEndCapture(handle, C.byref(graph))    # the refused call has ended the capture
        rt.cudaGetLastError()
        assert rc != 0
        torch.cuda.synchronize()
        for scale in (1.0, 2.0, 3.0):
            x.copy_(torch.from_numpy(h * scale))
            torch.cuda.synchronize()
            assert gpu_lib.hrn_vec_dot(s.h, x.numel(), p, p, C.byref(out)) == 0
            ref = float(np.dot(h * scale, h * scale))
            assert abs(out.value - ref) <= 1e-13 * ref
    for b in blocks[1::2]:
        assert rt.cudaFree(b) == 0

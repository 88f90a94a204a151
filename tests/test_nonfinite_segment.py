"""The reliable update after a segment of FP32 CG iterations that ended on a non-finite value: the
solution takes no increment (krylov.cu's dev_take_f32, called by its C++ name).  The values are
written by this test; nothing non-finite is computed on the way."""
import ctypes

import pytest

SC_STOP, SC_ALLOC = 24, 34
STOP_TEST, STOP_MAXIT, STOP_NONFINITE = 1, 2, 3


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 255, 70001])
@pytest.mark.parametrize("stop", [STOP_TEST, STOP_MAXIT, STOP_NONFINITE])
def test_increment_of_a_segment(gpulib, stop, n):
    import torch
    f = getattr(gpulib.load_library(), "_Z12dev_take_f32PdPfdxPKdP11CUstream_st")
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_double, ctypes.c_longlong,
                  ctypes.c_void_p, ctypes.c_void_p]
    g = torch.Generator().manual_seed(n)
    xh = torch.randn(n, generator=g)
    if stop == STOP_NONFINITE:
        xh[::3] = float("nan")
        xh[1::3] = float("inf")
    x = xh.cuda()
    y = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
    sc = torch.zeros(SC_ALLOC, dtype=torch.float64, device="cuda")
    sc[SC_STOP] = stop
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert f(y.data_ptr(), x.data_ptr(), 0.25, n, sc.data_ptr(), stream) == 0
    torch.cuda.synchronize()
    want = torch.zeros(n, dtype=torch.float64) if stop == STOP_NONFINITE else 0.25 * xh.double()
    assert torch.equal(y.cpu(), want)
    assert torch.equal(x.cpu(), torch.zeros(n))

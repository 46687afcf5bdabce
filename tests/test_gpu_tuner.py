"""The FP32 tile-shape tuner times only shapes that launch other kernels."""
import ctypes

import pytest

from test_gpu_parity import cube_setup

pytestmark = pytest.mark.gpu


def first_call_launches(s, shape=None):
    """kernels of a context's first FP32 matvec, with the tuner's, and of the second; the shape it ended with"""
    import torch

    import adda_gb300 as A
    c = A.Context(s.box, s.pos, s.mat, s.gridspace, s.wavenum, s.grid, nrhs_max=1)
    c.init_dmatrix()
    c.set_cc(0, s.cc[0].reshape(1, 3))
    default = list(c.fft_shape("fp32"))
    if shape:
        c.set_fft_shape(default, "fp32")
    x = torch.ones(3 * s.n, dtype=torch.complex64, device="cuda")
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    n = []
    for _ in range(2):
        before = A.kernel_launches()
        assert not c.L.adda_gb300_matvec_device(c.h, A.PREC["fp32"], 1, ctypes.c_void_p(x.data_ptr()),
                                                ctypes.c_void_p(y.data_ptr()), None, 0)
        n.append(A.kernel_launches() - before)
    torch.cuda.synchronize()
    got = list(c.fft_shape("fp32"))
    c.close()
    return n[0], n[1], default, got


# boxes whose matvec is one chunk whatever the tuner finds, x and z axes with radices above 16: the default and at most the
# three numbers of pairs are timed, not the 8, 32 z lines and 4 x lines that such axes have no kernels for
@pytest.mark.parametrize("box", [(100, 4, 100), (110, 4, 81)])
def test_no_shape_is_timed_twice(box):
    s = cube_setup(box, tuple(2 * b for b in box))
    first, one, default, got = first_call_launches(s)
    fixed = first_call_launches(s, True)[0]
    assert 1 <= (first - fixed) / (3 * one) <= 4
    assert got[:2] == default[:2]

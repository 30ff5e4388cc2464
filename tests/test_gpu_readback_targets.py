"""Readback into memory of any kind that a copy can reach: fresh host arrays,
pinned and managed ones, and device arrays, large and small."""
import ctypes

import numpy as np
import pytest

from taichi_lbm3d_gb300 import _native

pytestmark = pytest.mark.gpu


def targets(kind, n):
    import torch
    if kind == "device":
        t = torch.empty(n, device="cuda")
        return t, t.data_ptr(), lambda: t.cpu().numpy()
    if kind == "pinned":
        t = torch.empty(n, pin_memory=True)
        return t, t.data_ptr(), lambda: t.numpy()
    if kind == "read_before":            # pages in memory, with other contents
        a = np.full(n, 7.0, np.float32)
    else:
        a = np.empty(n, np.float32)
    return a, a.ctypes.data, lambda: a


@pytest.mark.parametrize("kind", ["fresh", "read_before", "pinned", "device"])
@pytest.mark.parametrize("shape", [(24, 20, 17), (160, 128, 130)])
def test_fields_into_any_memory(kind, shape):
    import torch
    solid = np.zeros(shape, np.int8)
    solid[2:5, 3:9, 4:7] = 1
    lat = _native.Lattice(_native.make_params(shape, niu=0.1, force=(1e-5, 0, 0), visc_convention=1, guo_convention=2))
    lat.set_geometry(solid)
    lat.init()
    lat.step(3)
    rho, v = lat.macros()
    n = int(np.prod(shape))
    (_r, pr, get_r), (_v, pv, get_v) = targets(kind, n), targets(kind, 3 * n)
    assert _native.load().lbm_get_macros(lat.h, ctypes.c_void_p(pr), ctypes.c_void_p(pv)) == 0
    torch.cuda.synchronize()
    assert np.array_equal(get_r(), rho.ravel(order="F"))
    assert np.array_equal(get_v(), v.reshape((n, 3), order="F").ravel())
    lat.close()


def test_batch_fields_into_device_memory():
    import torch
    from taichi_lbm3d_gb300.batch import Batch, _lib
    b = Batch([np.zeros((128, 128, 130), np.int8)], storage="f16")
    b.init()
    b.step(2, chunk=2)
    rho, v = b.macros(0)
    n = rho.size
    d, e = torch.empty(n, device="cuda"), torch.empty(3 * n, device="cuda")
    assert _lib().lbm_batch_get_macros(b.h, 0, ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(e.data_ptr())) == 0
    torch.cuda.synchronize()
    assert np.array_equal(d.cpu().numpy(), rho.ravel(order="F"))
    assert np.array_equal(e.cpu().numpy(), v.reshape((n, 3), order="F").ravel())
    b.close()

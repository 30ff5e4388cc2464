"""Steps taken while a caller captures another stream, in the same thread or another:
the caller's graph stays whole and the steps are the usual ones."""
import threading

import numpy as np
import pytest

from taichi_lbm3d_gb300 import _native
from taichi_lbm3d_gb300.geometry import sphere_pack

pytestmark = pytest.mark.gpu

SHAPE = (31, 26, 23)


def lattice():
    lat = _native.Lattice(_native.make_params(SHAPE, niu=0.1, force=(1e-5, 0, 0), visc_convention=1, guo_convention=2))
    lat.set_geometry(sphere_pack(SHAPE, 2.0, 4.0, 0.6, seed=11, percolate=False))
    lat.init()
    return lat


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
@pytest.mark.parametrize("other_thread", [False, True])
def test_steps_leave_a_callers_capture_alone(mode, other_thread):
    import torch
    lat = lattice()
    x = torch.zeros(256, device="cuda")
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=torch.cuda.Stream(), capture_error_mode=mode):
        x += 1
        if other_thread:
            t = threading.Thread(target=lat.step_async, args=(200,))
            t.start()
            t.join()
        else:
            lat.step_async(200)
        x += 1
    g.replay()
    torch.cuda.synchronize()
    assert x[0].item() == 2.0
    lat.synchronize()
    got = lat.macros()
    lat.close()
    ref = lattice()
    for _ in range(200):
        ref.step(1)
    assert all(np.array_equal(a, b) for a, b in zip(got, ref.macros()))
    ref.close()

"""Calls of a batch in other orders than configure, init, step."""
import numpy as np
import pytest

from taichi_lbm3d_gb300.geometry import sphere_pack

pytestmark = pytest.mark.gpu


def batch(storage="f32"):
    from taichi_lbm3d_gb300.batch import Batch
    return Batch([sphere_pack((24, 24, 24), 2, 4, 0.45, seed=51), sphere_pack((33, 20, 17), 2, 4, 0.45, seed=6)],
                 niu=0.1, force=(1e-5, 0, 0), storage=storage)


def fields(b):
    return b.macros(0) + b.macros(1)


@pytest.mark.parametrize("tile,block", [(64, 64), (32, 96), (96, 96), (256, 256)])
@pytest.mark.parametrize("use_graph", [True, False])
def test_configure_after_init_and_between_steps(tile, block, use_graph):
    """The tiles are cut for the CTA size that the steps are launched with."""
    b = batch()
    b.configure([tile] * 2, block)
    b.init()
    b.step(12, chunk=2, use_graph=use_graph)
    ref = fields(b)
    b.close()
    b = batch()
    b.init()
    b.configure([tile] * 2, block)
    b.step(4, chunk=2, use_graph=use_graph)
    b.configure([128] * 2, 128)
    b.step(4, chunk=2, use_graph=use_graph)
    b.configure([tile] * 2, block)
    b.step(4, chunk=2, use_graph=use_graph)
    assert all(np.array_equal(x, y) for x, y in zip(fields(b), ref))
    b.close()


@pytest.mark.parametrize("call", [lambda b: b.step(4, chunk=2), lambda b: b.step(4, chunk=2, use_graph=False),
                                  lambda b: b.run_to_convergence(check_every=2, max_steps=8)])
def test_steps_before_init_are_refused(call):
    """Without a state there is nothing to step; a zero Darcy velocity would read as converged."""
    from taichi_lbm3d_gb300 import _native
    b = batch()
    with pytest.raises(_native.LbmError):
        call(b)
    b.configure([64, 64], 64)
    b.init()
    call(b)
    b.close()


@pytest.mark.parametrize("storage", ["f32", "f16"])
def test_batch_without_any_fluid(storage):
    from taichi_lbm3d_gb300.batch import Batch
    b = Batch([np.ones((9, 7, 5), np.int8)], storage=storage)
    b.init()
    b.step(4, chunk=2)
    darcy, steps, conv = b.run_to_convergence(check_every=2, max_steps=8)
    rho, v = b.macros(0)
    b.close()
    assert darcy[0] == 0.0 and conv[0] and np.all(rho == 1.0) and np.all(v == 0.0)

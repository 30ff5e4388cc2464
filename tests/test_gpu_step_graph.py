"""Long runs of small lattices replay a captured run of steps; grouping the same
steps in any other way (single calls, odd splits that start from either buffer,
a new geometry or a new initial state in between) gives the same bits."""
import numpy as np
import pytest

from taichi_lbm3d_gb300 import _native
from taichi_lbm3d_gb300.geometry import sphere_pack

pytestmark = pytest.mark.gpu

SHAPE = (31, 26, 23)


def lattice(kind, solid):
    kw = dict(niu=0.1, force=(1e-5, 0.0, 0.0), visc_convention=1, guo_convention=1)
    if kind == "two_phase":
        kw.update(two_phase=True, bc_form=1, psi_bc=(1, 1, 0, 0, 0, 0), psi_val=(1.0, -1.0, 1, 1, 1, 1))
    if kind == "f64":
        kw.update(storage="f64")
    lat = _native.Lattice(_native.make_params(SHAPE, **kw))
    lat.set_geometry(solid)
    if kind == "two_phase":
        psi = -np.ones(SHAPE, np.float32)
        psi[:5] = 1.0
        lat.set_psi(psi)
    if kind == "grey":
        lat.set_grey(np.where(solid > 0, 1.0, 0.2))
    lat.init()
    return lat


def fields(lat, kind):
    return list(lat.macros()) + (list(lat.phase()) if kind == "two_phase" else [])


@pytest.mark.parametrize("kind", ["f32", "f64", "grey", "two_phase"])
def test_grouping_does_not_change_the_result(kind):
    solid = sphere_pack(SHAPE, 2.0, 4.0, 0.6, seed=11, percolate=False)
    res = []
    for groups in ([200], [1] * 200, [33, 1, 130, 36], [129, 71]):
        lat = lattice(kind, solid)
        for n in groups:
            lat.step(n)
        res.append(fields(lat, kind))
        lat.close()
    assert all(np.isfinite(x).all() for x in res[0]) and np.abs(res[0][1]).max() > 0
    for r in res[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(res[0], r))


def test_new_state_and_new_geometry_after_a_replayed_run():
    solid = sphere_pack(SHAPE, 2.0, 4.0, 0.6, seed=11, percolate=False)
    other = sphere_pack(SHAPE, 2.0, 4.0, 0.5, seed=12, percolate=False)
    lat = lattice("f32", solid)
    lat.step(201)
    lat.init()
    lat.step(150)
    again = fields(lat, "f32")
    lat.set_geometry(other)
    lat.init()
    lat.step(150)
    moved = fields(lat, "f32")
    lat.close()
    for mask, got in ((solid, again), (other, moved)):
        ref = lattice("f32", mask)
        for _ in range(150):
            ref.step(1)
        assert all(np.array_equal(a, b) for a, b in zip(fields(ref, "f32"), got))
        ref.close()

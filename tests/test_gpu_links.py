"""Neighbour links (csrc/lbm_links.cuh) at the edges of their encoding: group
remainders, lattices that are all periodic seam, rows that leave the 5-bit
distance (with and without room in the first record allocation).  FP32
reference arithmetic, bit for bit against the oracle: a wrong source cannot
go unseen."""
import numpy as np
import pytest

from oracle.oracle import Oracle, make_params as oracle_params
from taichi_lbm3d_gb300 import _native

pytestmark = pytest.mark.gpu


def check(p, solid, steps):
    o = Oracle(p, solid)
    o.step(steps)
    lat = _native.Lattice(_native.make_params(
        (p.nx, p.ny, p.nz), niu=p.niu, force=tuple(p.force), bc=tuple(p.bc), rho_bc=tuple(p.rho_bc),
        vel_bc=[tuple(v) for v in p.vel_bc], visc_convention=p.visc_convention, guo_convention=p.guo_convention,
        bc_form=p.bc_form))
    lat.set_geometry(solid)
    lat.init()
    lat.step(steps)
    rho, v = lat.macros()
    lat.close()
    fl = solid == 0
    assert np.array_equal(rho[fl], o.field("rho").astype(np.float32)[fl])
    assert np.array_equal(v[fl], o.field("v").astype(np.float32)[fl])


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 127, 129])
def test_group_remainders_on_a_seam_only_lattice(n):
    p = oracle_params((n, 1, 1), niu=0.1, force=(1e-5, 2e-5, -1e-5), visc_convention=1, guo_convention=2)
    check(p, np.zeros((n, 1, 1), np.int8), 7)


@pytest.mark.parametrize("bc,bc_form", [((0,) * 6, 0), ((1,) * 6, 0), ((1, 0, 2, 2, 0, 1), 0), ((2, 1, 0, 0, 2, 0), 1)])
def test_rows_out_of_the_distance_range(bc, bc_form):
    """Sparse planes between full ones: a group's 32 nodes face five times as many."""
    shape = (41, 37, 9)
    solid = np.zeros(shape, np.int8)
    i, j, k = np.indices(shape)
    solid[(k % 2 == 0) & ((i + 3 * j) % 5 != 0)] = 1
    p = oracle_params(shape, niu=0.1, bc=bc, rho_bc=(1.001, 1.0, 1.0005, 1.0, 1.0, 0.9995),
                      vel_bc=((1e-3, 0, 0), (0, 0, 1e-3), (0, 5e-4, 0), (0, 0, 0), (0, 0, 2e-4), (0, 0, 0)), bc_form=bc_form)
    check(p, solid, 20)

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


@pytest.mark.parametrize("shape,bc,psi_bc", [
    ((41, 37, 9), (0,) * 6, (0,) * 6),                     # rows out of range, all seams periodic
    ((41, 37, 9), (1, 1, 0, 0, 2, 0), (1, 0, 0, 1, 0, 0)),  # faces without a constant psi and the reverse
    ((33, 1, 3), (0,) * 6, (1, 1, 0, 0, 0, 0)),            # one cell thin
    ((130, 3, 2), (1, 2, 0, 0, 0, 0), (0, 0, 1, 0, 0, 1)),
])
def test_two_phase_links_match_oracle(shape, bc, psi_bc):
    rng = np.random.default_rng(5)
    i, j, k = np.indices(shape)
    solid = ((k % 2 == 0) & ((i + 3 * j) % 5 != 0)).astype(np.int8) if shape[2] == 9 else \
        (rng.random(shape) < 0.2).astype(np.int8)
    psi0 = np.where(i < shape[0] // 3, 1.0, -1.0).astype(np.float32)
    kw = dict(force=(5e-5, -2e-5, 1e-5), bc=bc, rho_bc=(1.001, 1.0, 1.0, 1.0, 1.0, 1.0), bc_form=1, two_phase=True,
              niu_l=0.05, niu_g=0.2, psi_solid=0.7, cap_a=0.005, psi_bc=psi_bc, psi_val=(1.0, -1.0, 0.5, 1.0, -1.0, -0.5))
    o = Oracle(oracle_params(shape, niu=0.1, visc_convention=1, guo_convention=1, **kw), solid, psi0)
    o.step(15)
    lat = _native.Lattice(_native.make_params(shape, niu=0.1, visc_convention=1, guo_convention=1, **kw))
    lat.set_geometry(solid)
    lat.set_psi(psi0)
    lat.init()
    lat.step(7)      # v of the seventh step is kept where a pressure face needs it, the rest is written by the last
    lat.step(8)
    rho, v = lat.macros()
    got = dict(zip(("psi", "rho_r", "rho_b"), lat.phase()), rho=rho, v=v)
    lat.close()
    fl = solid == 0
    for f, g in got.items():
        assert np.array_equal(g[fl], o.field(f).astype(np.float32)[fl]), f
    assert np.array_equal(got["psi"][~fl], psi0[~fl])

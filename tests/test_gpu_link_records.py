"""A node finds its own record of explicit links (csrc/lbm_linkgather.cuh) whichever
lanes of its warp run together, and lattices whose last group of 32 is partial
stream as the oracle does."""
import ctypes

import numpy as np
import pytest

from oracle.oracle import Oracle, make_params as oracle_params
from taichi_lbm3d_gb300 import _native
from tests.device_code import compile_device

pytestmark = pytest.mark.gpu

SRC = r"""
#include <cuda_runtime.h>
#include "lbm_kernels.cuh"
#include "lbm_linkgather.cuh"
using namespace lbmk;
// record index of every node that has one, the lanes split over two branches
__global__ void index_kernel(LbmLinks L, int split, int* out) {
    const int n = blockIdx.x * 32 + threadIdx.x;
    NodeLinks K;
    if (n % split == 0) {
        K.load(L, n);
        if (K.bits & LBM_LINK_EXC) out[n] = (int)((K.record(L) - L.rec) / LBM_LINK_REC);
        __threadfence();
    } else {
        __nanosleep(200);
        K.load(L, n);
        if (K.bits & LBM_LINK_EXC) out[n] = (int)((K.record(L) - L.rec) / LBM_LINK_REC);
    }
}
extern "C" int record_index(const void* node, const void* head, const void* recs, int groups, int split, int* out) {
    const LbmLinks L{(const uint2*)node, (const LbmLinkHead*)head, (const LbmLinkRecs*)recs, nullptr};
    index_kernel<<<groups, 32>>>(L, split, out);
    return cudaDeviceSynchronize();
}
"""


def test_record_index_of_split_warps(tmp_path):
    import torch
    lib = compile_device(tmp_path, "records", SRC)
    rng = np.random.default_rng(4)
    groups = 7
    has = rng.random((groups, 32)) < np.array([0.0, 0.1, 0.5, 0.5, 0.9, 1.0, 1.0])[:, None]
    node = np.zeros((groups * 32, 2), np.uint32)
    node[:, 1] = has.ravel()
    first = np.concatenate([[0], np.cumsum(has.sum(1))[:-1]])
    recs = np.stack([first, (has * (1 << np.arange(32, dtype=np.int64))).sum(1)], 1).astype(np.uint32)
    ref = np.where(has, first[:, None] + np.cumsum(has, 1) - 1, -1).ravel()
    dev = [torch.from_numpy(a.view(np.int32)).cuda() for a in (node, np.zeros((groups, 8), np.uint32), recs)]
    for split in (2, 3, 5, 33):
        out = torch.full((groups * 32,), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert lib.record_index(*[ctypes.c_void_p(t.data_ptr()) for t in dev], groups, split,
                                ctypes.c_void_p(out.data_ptr())) == 0
        assert np.array_equal(out.cpu().numpy(), ref), split


@pytest.mark.parametrize("n", [1, 2, 5, 31, 32, 33, 47, 63, 64, 65])
@pytest.mark.parametrize("two_phase", [False, True])
def test_partial_last_group(n, two_phase):
    shape = (n, 1, 2)
    kw = dict(force=(5e-5, -2e-5, 1e-5))
    psi = None
    if two_phase:
        kw.update(bc_form=1, two_phase=True, niu_l=0.05, niu_g=0.2, psi_solid=0.7, cap_a=0.005)
        psi = np.where(np.arange(n) < (n + 1) // 2, 1.0, -1.0).astype(np.float32)[:, None, None] * np.ones(shape, np.float32)
    solid = np.zeros(shape, np.int8)
    solid[n // 2, 0, 0] = n > 2
    o = Oracle(oracle_params(shape, niu=0.1, visc_convention=1, guo_convention=1, **kw), solid, psi)
    o.step(9)
    lat = _native.Lattice(_native.make_params(shape, niu=0.1, visc_convention=1, guo_convention=1, **kw))
    lat.set_geometry(solid)
    if two_phase:
        lat.set_psi(psi)
    lat.init()
    lat.step(9)
    got = dict(zip(("rho", "v"), lat.macros()))
    if two_phase:
        got.update(zip(("psi", "rho_r", "rho_b"), lat.phase()))
    lat.close()
    fl = solid == 0
    for f, g in got.items():
        assert np.array_equal(g[fl], o.field(f).astype(np.float32)[fl], equal_nan=True), f


@pytest.mark.parametrize("shape", [(70, 9, 1), (9, 70, 1), (33, 1, 5), (40, 37, 2), (5, 7, 3), (16, 8, 8), (24, 6, 9),
                                   (1, 9, 9), (2, 5, 5), (1, 1, 40)])
@pytest.mark.parametrize("bc,bc_form", [((0,) * 6, 0), ((0, 0, 1, 0, 0, 0), 0), ((0, 0, 0, 2, 0, 0), 1),
                                        ((1, 1, 0, 0, 0, 0), 0), ((0, 0, 0, 0, 2, 1), 0)])
@pytest.mark.parametrize("dense", [0.0, 0.3])
def test_rows_across_seams(shape, bc, bc_form, dense):
    """Rows across periodic y and z faces, alone and beside fixed faces, bit for bit."""
    if any(bc[f] and shape[f // 2] < 2 for f in range(6)):
        pytest.skip("a fixed face needs two cells")
    solid = (np.random.default_rng(7).random(shape) < dense).astype(np.int8)
    kw = dict(niu=0.1, force=(1e-4, -2e-4, 1e-4), bc=bc, rho_bc=(1.002, 1.0, 1.001, 1.0, 1.0, 0.999),
              vel_bc=((0, 0, 0), (0, 0, 0), (0, 0, 0), (1e-3, 0, 2e-3), (2e-3, 1e-3, 0), (0, 0, 0)), bc_form=bc_form,
              visc_convention=1, guo_convention=2)
    o = Oracle(oracle_params(shape, **kw), solid)
    o.step(12)
    lat = _native.Lattice(_native.make_params(shape, **kw))
    lat.set_geometry(solid)
    lat.init()
    lat.step(12)
    fl = solid == 0
    for f, g in zip(("rho", "v"), lat.macros()):
        assert np.array_equal(g[fl], o.field(f).astype(np.float32)[fl]), f
    lat.close()


@pytest.mark.parametrize("shape", [(512, 256, 1), (256, 64, 4)])
def test_flat_lattices_need_few_records(shape):
    """Only nodes of the x faces, and where a row starts anew, hold explicit links: 180 B of
    populations and fields a node, 17 B of index and links, and no 80 B record each."""
    lat = _native.Lattice(_native.make_params(shape, niu=0.1))
    lat.set_geometry(np.zeros(shape, np.int8))
    per_node = lat.info().device_bytes / np.prod(shape)
    lat.close()
    assert per_node < 205

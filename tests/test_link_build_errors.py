"""A failed build of the neighbour links leaves none behind: a handle that kept
half-built ones would take them for finished at its next use.  The CUDA calls are
stand-ins whose k-th one fails; no GPU."""
import ctypes
import subprocess

import pytest

SRC = r"""
#include <cuda_runtime.h>
#include <cstdlib>
static int g_call, g_fail, g_live;
static cudaError_t step() { return g_call++ == g_fail ? cudaErrorUnknown : cudaSuccess; }
static cudaError_t f_malloc(void** p, size_t) { if (step() != cudaSuccess) return cudaErrorMemoryAllocation; *p = std::malloc(64); ++g_live; return cudaSuccess; }
static cudaError_t f_free(void* p) { if (p) --g_live; std::free(p); return cudaSuccess; }
#define cudaMalloc(p, n) f_malloc((void**)(p), n)
#define cudaFree(p) f_free((void*)(p))
#define cudaMemsetAsync(...) step()
#define cudaMemcpyAsync(...) step()
#define cudaStreamSynchronize(...) step()
#define cudaGetLastError() step()
#include "lbm_links.cu"
int lbm_cuda_check(LbmHandle*, cudaError_t e, const char*) { return e == cudaSuccess ? LBM_OK : LBM_ECUDA; }
extern "C" int run(int fail, int* kept, long long* bytes, int* live) {
    g_call = g_live = 0;
    g_fail = fail;
    LbmHandle h;
    h.p = LbmParams();
    h.np = 0;                                     // no fluid, no groups: nothing is launched
    const LbmLinkLattice lat{8, 4, 2, 0, 0, 0};
    const int rc = links_build(&h, &lat, 1);
    *kept = h.d_links != nullptr;
    *bytes = h.device_bytes;
    *live = g_live;
    if (h.d_links) f_free(h.d_links);
    h.d_links = nullptr;
    return rc;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    import os
    import shutil
    from taichi_lbm3d_gb300 import build
    nvcc = build._nvcc()
    if shutil.which(nvcc) is None and not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    d = tmp_path_factory.mktemp("links")
    cu, so = str(d / "links.cu"), str(d / "links.so")
    with open(cu, "w") as fh:
        fh.write(SRC)
    r = subprocess.run([nvcc] + build.NVCC_FLAGS + ["-I", build.CSRC, "-shared", cu, "-o", so], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return ctypes.CDLL(so)


@pytest.mark.parametrize("fail", [-1, 0, 1, 2, 3, 4])
def test_nothing_is_kept_of_a_failed_build(lib, fail):
    kept, nbytes, live = ctypes.c_int(), ctypes.c_longlong(), ctypes.c_int()
    rc = lib.run(fail, ctypes.byref(kept), ctypes.byref(nbytes), ctypes.byref(live))
    if fail < 0:
        assert rc == 0 and kept.value == 1 and nbytes.value > 0 and live.value == 1
    else:
        assert rc != 0 and (kept.value, nbytes.value, live.value) == (0, 0, 0)

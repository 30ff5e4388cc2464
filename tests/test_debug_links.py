"""The -DLBM_DEBUG build steps each storage with the kernel of the default build,
its index checks compiled in: the neighbour links, and the map for FP64.
Compile-only: no GPU."""
import os
import shutil
import subprocess

import pytest

from taichi_lbm3d_gb300 import build


def kernels(obj):
    out = subprocess.run(["nm", "-C", obj], capture_output=True, text=True, check=True).stdout
    return {k: any(k in line for line in out.splitlines()) for k in ("sp_link_kernel", "sp_step_kernel")}


def test_debug_build_keeps_the_link_kernel(tmp_path):
    nvcc = build._nvcc()
    if shutil.which("nm") is None or (shutil.which(nvcc) is None and not os.path.exists(nvcc)):
        pytest.skip("nvcc or nm not available")
    obj = str(tmp_path / "sp.o")
    r = subprocess.run([nvcc] + build.NVCC_FLAGS + ["-DLBM_DEBUG", "-c", os.path.join(build.CSRC, "lbm_sp.cu"), "-o", obj],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert kernels(obj) == {"sp_link_kernel": True, "sp_step_kernel": True}


def test_every_gathered_link_is_checked():
    """No population is loaded from a decoded source that has not gone through the check."""
    txt = open(os.path.join(build.CSRC, "lbm_linkgather.cuh")).read()
    body = txt[txt.index("struct LinkGather"):]
    assert body.count("checked(") == 3 and "lbm_eoff32(K." not in body and "lbm_eoff32(SRC)" not in body

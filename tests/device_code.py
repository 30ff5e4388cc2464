"""Builds a few lines of device code against the library's own headers."""
import ctypes
import subprocess


def compile_device(tmp_path, name, src):
    """The shared library of `src` (CUDA C++ with extern "C" launchers), with the library's flags."""
    from taichi_lbm3d_gb300 import build
    cu, so = str(tmp_path / (name + ".cu")), str(tmp_path / (name + ".so"))
    with open(cu, "w") as fh:
        fh.write(src)
    r = subprocess.run([build._nvcc()] + build.NVCC_FLAGS + ["-I", build.CSRC, "-shared", cu, "-o", so],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return ctypes.CDLL(so)

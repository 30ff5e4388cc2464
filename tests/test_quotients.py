"""The quotients of the step kernels (csrc/lbm_kernels.cuh): product with a
correctly rounded reciprocal and one fused residual correction equal the IEEE
quotient, for the divisors 3 and 9 at every FP32 significand and for random
densities."""
import ctypes
import ctypes.util

import numpy as np
import pytest

F = np.float32


@pytest.mark.parametrize("n", [3, 9])
def test_constant_divisors_every_significand(n):
    a = np.arange(1 << 23, 1 << 24, dtype=np.uint32).astype(F)      # all significands; powers of two only scale
    y = F(1.0 / n)
    q = a * y
    # a - n q is a small multiple of ulp(a), so FP64 holds it and the corrected quotient exactly
    res = (a.astype(np.float64) - float(n) * q.astype(np.float64)).astype(F)
    got = (res.astype(np.float64) * float(y) + q.astype(np.float64)).astype(F)
    assert np.array_equal(got, a / F(n))


def test_reciprocal_with_residual_equals_division():
    libm = ctypes.CDLL(ctypes.util.find_library("m") or "libm.so.6")
    libm.fmaf.argtypes = [ctypes.c_float] * 3
    libm.fmaf.restype = ctypes.c_float
    rng = np.random.default_rng(3)
    a = (rng.standard_normal(60000) * 10.0 ** rng.uniform(-9, 0, 60000)).astype(F)
    b = np.concatenate([1 + 1e-3 * rng.standard_normal(30000), 10.0 ** rng.uniform(-5.9, 5.9, 30000)]).astype(F)
    y = (1.0 / b.astype(np.float64)).astype(F)                       # correctly rounded reciprocal (FP64 has 2 x 24 + 2 bits)
    for x, d, r in zip(a.tolist(), b.tolist(), y.tolist()):
        q = float(F(x) * F(r))
        got = libm.fmaf(libm.fmaf(q, -d, x), r, q)
        assert F(got) == F(x) / F(d), (x, d)

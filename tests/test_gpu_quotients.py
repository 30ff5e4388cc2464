"""The quotients that the step kernels share a reciprocal for (csrc/lbm_kernels.cuh),
run on the GPU: the division bit for bit, but for numerators below 2^-60 (a unit
in the last place) and finite ones above 2^80."""
import ctypes

import numpy as np
import pytest

from tests.device_code import compile_device

pytestmark = pytest.mark.gpu

SRC = r"""
#include <cuda_runtime.h>
#include "lbm_kernels.cuh"
using namespace lbmk;
__device__ bool same(float x, float y) {
    return __float_as_uint(x) == __float_as_uint(y) || (x != x && y != y);
}
__global__ void const_kernel(unsigned long long* bad) {
    unsigned long long n = 0;
    for (unsigned long long u = blockIdx.x * blockDim.x + threadIdx.x; u < 1ull << 32; u += gridDim.x * blockDim.x) {
        const float a = __uint_as_float((uint32_t)u);
        n += !same(div_const<3>(a), a / 3.0f) + !same(div_const<9>(a), a / 9.0f);
    }
    if (n) atomicAdd(bad, n);
}
template <int K>
__global__ void quot_kernel(const float* a, const float* b, int n, unsigned long long* bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float x[K];
    for (int k = 0; k < K; ++k) x[k] = a[(int64_t)k * n + i];
    quotients(x, b[i]);
    unsigned long long m = 0;
    for (int k = 0; k < K; ++k) {
        const float num = a[(int64_t)k * n + i], ref = num / b[i];
        const bool tiny = fabsf(num) < 0x1p-60f, huge = fabsf(num) >= 0x1p80f && !isinf(num);
        const int ulps = (int)(__float_as_uint(x[k]) - __float_as_uint(ref));
        m += !(same(x[k], ref) || (tiny && num != 0.0f && abs(ulps) <= 1) || huge);
    }
    if (m) atomicAdd(bad, m);
}
template <int FORCE>
__global__ void guo_kernel(const float* v, const float* f, int n, int guo, unsigned long long* bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float vx = v[i], vy = v[n + i], vz = v[2 * n + i];
    const float fe[3] = {f[i], FORCE == FORCE_X ? 0.0f : f[n + i], FORCE == FORCE_X ? 0.0f : f[2 * n + i]};
    float G[19];
    guo_dense<float, FORCE>(G, vx, vy, vz, fe, guo);
    unsigned long long m = 0;
#define ONE(S) {                                                                                          \
        float a = ((float)lbm_ex(S) - vx) * fe[0], ee = lbm_edot<S, float>(vx, vy, vz);                    \
        if (FORCE != FORCE_X) a = a + ((float)lbm_ey(S) - vy) * fe[1];                                     \
        if (FORCE != FORCE_X) a = a + ((float)lbm_ez(S) - vz) * fe[2];                                     \
        if (FORCE == FORCE_X) ee = lbm_ex(S) == 0 ? 0.0f : ee * ((float)lbm_ex(S) * fe[0]);                \
        else ee = ee * lbm_edot<S, float>(fe[0], fe[1], fe[2]);                                            \
        const float g = guo == 0 ? a / 3.0f + ee / 9.0f : guo == 1 ? a + ee : 3.0f * a + 9.0f * ee;        \
        m += !same(G[S], (float)lbm_w(S) * g);                                                             \
    }
    ONE(0) LBM_ALL_DIRS(ONE)
    if (m) atomicAdd(bad, m);
}
extern "C" int run_const(unsigned long long* bad) {
    const_kernel<<<2432, 256>>>(bad);
    return cudaDeviceSynchronize();
}
extern "C" int run_quot(const float* a, const float* b, int n, int k, unsigned long long* bad) {
    if (k == 1) quot_kernel<1><<<(n + 255) / 256, 256>>>(a, b, n, bad);
    if (k == 4) quot_kernel<4><<<(n + 255) / 256, 256>>>(a, b, n, bad);
    if (k == 6) quot_kernel<6><<<(n + 255) / 256, 256>>>(a, b, n, bad);
    if (k == 12) quot_kernel<12><<<(n + 255) / 256, 256>>>(a, b, n, bad);
    return cudaDeviceSynchronize();
}
extern "C" int run_guo(const float* v, const float* f, int n, int guo, int x, unsigned long long* bad) {
    if (x) guo_kernel<FORCE_X><<<(n + 255) / 256, 256>>>(v, f, n, guo, bad);
    else guo_kernel<FORCE_ANY><<<(n + 255) / 256, 256>>>(v, f, n, guo, bad);
    return cudaDeviceSynchronize();
}
"""

N = 1 << 21
EDGE = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, -1e-45, 1.1754944e-38, 3.4028235e38, 1.0, 2.0 ** -60, 2.0 ** 80,
                 2.0 ** -40, 2.0 ** 40], np.float32)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return compile_device(tmp_path_factory.mktemp("quot"), "quotients", SRC)


def bits(rng, n):
    return rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32).view(np.float32)


def scaled(rng, n, lo, hi):
    return (rng.choice([-1.0, 1.0], n) * rng.uniform(1, 2, n) * 2.0 ** rng.uniform(lo, hi, n)).astype(np.float32)


def mixed(rng, n):
    """Zeros, infinities, NaN, subnormals and the bounds of the rule among ordinary numbers."""
    x = np.where(rng.random(n) < 0.3, rng.choice(np.concatenate([EDGE, np.nextafter(EDGE, np.float32(0)),
                                                                  np.nextafter(EDGE, np.float32(np.inf))]), n),
                 scaled(rng, n, -8, 1))
    return x.astype(np.float32)


KINDS = {
    "flow": (lambda r, n: scaled(r, n, -40, 0), lambda r, n: (1 + 1e-2 * r.standard_normal(n)).astype(np.float32)),
    "stored_fp16_scale": (lambda r, n: scaled(r, n, -24, 17), lambda r, n: (65536 * (1 + 1e-2 * r.standard_normal(n))).astype(np.float32)),
    "whole_divisor_range": (lambda r, n: scaled(r, n, -62, 82), lambda r, n: np.abs(scaled(r, n, -42, 42))),
    "any_patterns": (bits, bits),
    "edges": (mixed, mixed),
}


def run(call):
    import torch
    bad = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    assert call(ctypes.c_void_p(bad.data_ptr())) == 0
    return int(bad.item())


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def test_constant_divisors_every_number(lib):
    assert run(lib.run_const) == 0


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("k", [1, 4, 6, 12])
def test_shared_reciprocal_is_the_division(lib, kind, k):
    rng = np.random.default_rng(k)
    n = N // k
    with np.errstate(all="ignore"):
        a, b = dev(np.stack([KINDS[kind][0](rng, n) for _ in range(k)])), dev(KINDS[kind][1](rng, n))
    assert run(lambda bad: lib.run_quot(ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(b.data_ptr()), n, k, bad)) == 0


@pytest.mark.parametrize("kind", ["flow", "any_patterns", "edges"])
@pytest.mark.parametrize("guo", [0, 1, 2])
@pytest.mark.parametrize("x_only", [0, 1])
def test_guo_terms_are_the_divided_ones(lib, kind, guo, x_only):
    rng = np.random.default_rng(guo)
    n = N // 8
    with np.errstate(all="ignore"):
        v = dev(np.stack([KINDS[kind][0](rng, n) for _ in range(3)]))
        f = scaled(rng, 3 * n, -20, -3) if kind == "flow" else KINDS[kind][0](rng, 3 * n)
    f = dev(f.reshape(3, n))
    assert run(lambda bad: lib.run_guo(ctypes.c_void_p(v.data_ptr()), ctypes.c_void_p(f.data_ptr()), n, guo, x_only, bad)) == 0

"""Weight gradient where a CTA runs through its buffers several times: 6,348 blocks of
8 x 4 x 4 voxels, six a CTA (two buffers of input halo and g, each loaded three times),
ragged in every axis, against FP64."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout", [(16, 16), (48, 16), (32, 32), (64, 64), (32, 64)])
def test_weight_gradient_over_many_blocks(cin, cout):
    import torch
    from taichi_lbm3d_gb300 import unet
    L = unet._lib()
    n, d, h, w = 1, 89, 91, 93
    gen = torch.Generator(device="cuda").manual_seed(cin + cout)
    x = torch.randn(n, d, h, w, cin, generator=gen, device="cuda").to(torch.bfloat16)
    g = torch.randn(n, d, h, w, cout, generator=gen, device="cuda").to(torch.bfloat16)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    scr = torch.full((int(L.lbm_nn_wgrad_scratch_floats(n, d, h, w, cin, cout)),), float("nan"), device="cuda")
    runs = []
    for _ in range(3):
        dw = torch.full((cout, 27, cin), float("nan"), device="cuda")
        db = torch.full((cout,), float("nan"), device="cuda")
        assert L.lbm_nn_conv3d_wgrad(p(x), p(g), p(dw), p(db), p(scr), scr.numel(), n, d, h, w, cin, cout, s) == 0
        torch.cuda.synchronize()
        runs.append((dw, db))
    flag = ctypes.c_int(0)
    assert L.lbm_nn_tc_status(ctypes.byref(flag)) == 0 and flag.value == 0
    dw, db = runs[0]
    assert all(torch.equal(a, dw) and torch.equal(b, db) for a, b in runs[1:])

    xp = torch.zeros(n, d + 2, h + 2, w + 2, cin, dtype=torch.float64, device="cuda")
    xp[:, 1:-1, 1:-1, 1:-1] = x.double()
    g64 = g.double().reshape(-1, cout)
    # products of bf16 are exact in FP32; a sum of V terms in any order is off by at most
    # (V - 1) 2^-24 of the terms' sizes, in practice sqrt(V) of it; four times that, with truncating adds
    bar = 4 * np.sqrt(g64.shape[0]) * 2.0 ** -24
    for t in range(27):
        kz, ky, kx = t // 9, t // 3 % 3, t % 3
        xs = xp[:, kz:kz + d, ky:ky + h, kx:kx + w].reshape(-1, cin)
        assert ((dw[:, t].double() - g64.T @ xs).abs() <= bar * (g64.abs().T @ xs.abs())).all(), t
    assert ((db.double() - g64.sum(0)).abs() <= bar * g64.abs().sum(0)).all()

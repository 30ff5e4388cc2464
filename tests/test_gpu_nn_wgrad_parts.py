"""Weight gradient in parts of 16 input channels against FP64, on both sides of the rule."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# volumes: less than one 8 x 4 x 4 block, ragged in every axis, more blocks than CTAs of a part hold
@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 16), (32, 32), (48, 32), (64, 16), (64, 32), (80, 32), (96, 16),
                                      (128, 32)])
@pytest.mark.parametrize("dims", [(1, 2, 3, 5), (2, 5, 9, 17), (1, 17, 23, 41)])
def test_weight_gradient_in_parts(cin, cout, dims):
    import torch
    from taichi_lbm3d_gb300 import unet
    L = unet._lib()
    n, d, h, w = dims
    torch.manual_seed(cin + cout)
    x = torch.randn(n, d, h, w, cin).to(torch.bfloat16)
    g = torch.randn(n, d, h, w, cout).to(torch.bfloat16)
    xg, gg = x.cuda(), g.cuda()
    dw = torch.full((cout, 27, cin), float("nan"), device="cuda")
    db = torch.full((cout,), float("nan"), device="cuda")
    scr = torch.empty(int(L.lbm_nn_wgrad_scratch_floats(n, d, h, w, cin, cout)), device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.lbm_nn_conv3d_wgrad(p(xg), p(gg), p(dw), p(db), p(scr), scr.numel(), n, d, h, w, cin, cout, s) == 0
    torch.cuda.synchronize()
    flag = ctypes.c_int(0)
    assert L.lbm_nn_tc_status(ctypes.byref(flag)) == 0 and flag.value == 0

    xp = np.zeros((n, d + 2, h + 2, w + 2, cin))
    xp[:, 1:-1, 1:-1, 1:-1] = x.float().numpy()
    g64 = g.double().numpy().reshape(-1, cout)
    ref, size = np.empty((cout, 27, cin)), np.empty((cout, 27, cin))
    for t in range(27):
        kz, ky, kx = t // 9, t // 3 % 3, t % 3
        xs = xp[:, kz:kz + d, ky:ky + h, kx:kx + w].reshape(-1, cin)
        ref[:, t], size[:, t] = g64.T @ xs, np.abs(g64).T @ np.abs(xs)
    # products of bf16 are exact in FP32; a sum of V terms in any order is off by at most
    # (V - 1) 2^-24 of the terms' sizes, in practice sqrt(V) of it; twice that for truncating adds
    v = g64.shape[0]
    bar = 4 * np.sqrt(v) * 2.0 ** -24
    assert (np.abs(dw.cpu().numpy() - ref) <= bar * size + 1e-30).all()
    assert (np.abs(db.cpu().numpy() - g64.sum(0)) <= bar * np.abs(g64).sum(0) + 1e-30).all()

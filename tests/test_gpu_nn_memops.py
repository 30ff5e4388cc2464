"""The U-Net's memory kernels (pool, upsample, concat, split and their
backward passes) run as 16-byte vectors when channel counts are multiples of 8
and the tensors are 16-byte aligned, else element by element.  Both forms do
the same per-element arithmetic in the same order, so a call on aligned
tensors must equal, bit for bit, the same call on tensors shifted by one BF16
element (which takes the element form).  The one-pass head weight gradient
(16 -> 4) is checked against FP64 and against its general form."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, D, H, W = 1, 6, 8, 10


def _lib():
    from taichi_lbm3d_gb300 import unet
    return unet._lib()


def _pair(t, shape, dtype):
    """The same values twice: an aligned tensor and a view one element past a 16-byte boundary."""
    import torch
    n = int(np.prod(shape))
    a = t.reshape(shape).to(dtype).contiguous().cuda()
    buf = torch.zeros(n + 1, dtype=dtype, device="cuda")
    buf[1:] = a.reshape(-1)
    return a, buf[1:].view(shape)


def _p(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _s():
    import torch
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _same(x, y):
    import torch
    torch.cuda.synchronize()
    assert torch.equal(x.view(torch.int16) if x.dtype == torch.bfloat16 else x,
                       y.view(torch.int16) if y.dtype == torch.bfloat16 else y)


@pytest.mark.parametrize("c", [16, 48])
def test_pool_and_its_gradient_vector_equals_elementwise(c):
    import torch
    L = _lib()
    torch.manual_seed(c)
    x = torch.randn(N, D, H, W, c)
    xa, xu = _pair(x, (N, D, H, W, c), torch.bfloat16)
    oa = torch.empty(N, D // 2, H // 2, W // 2, c, dtype=torch.bfloat16, device="cuda")
    ou = torch.zeros((oa.numel() + 1,), dtype=torch.bfloat16, device="cuda")[1:].view(oa.shape)
    aa = torch.empty(oa.shape, dtype=torch.uint8, device="cuda")
    au = torch.zeros((oa.numel() + 1,), dtype=torch.uint8, device="cuda")[1:].view(oa.shape)
    assert L.lbm_nn_pool2(_p(xa), _p(oa), _p(aa), N, D, H, W, c, _s()) == 0
    assert L.lbm_nn_pool2(_p(xu), _p(ou), _p(au), N, D, H, W, c, _s()) == 0
    _same(oa, ou)
    _same(aa, au)
    g = torch.randn(oa.shape)
    ga, gu = _pair(g, oa.shape, torch.bfloat16)
    m = torch.randn(N, D, H, W, c)
    ma, mu = _pair(m, (N, D, H, W, c), torch.bfloat16)
    prev = torch.randn(N, D, H, W, c)
    for acc in (0, 1):
        ia, iu = _pair(prev, (N, D, H, W, c), torch.bfloat16)
        assert L.lbm_nn_pool2_bwd(_p(ga), _p(aa), _p(ia), _p(ma), N, D, H, W, c, acc, _s()) == 0
        assert L.lbm_nn_pool2_bwd(_p(gu), _p(au), _p(iu), _p(mu), N, D, H, W, c, acc, _s()) == 0
        _same(ia, iu)


@pytest.mark.parametrize("c", [16, 64])
def test_upsample_and_its_gradient_vector_equals_elementwise(c):
    import torch
    L = _lib()
    torch.manual_seed(c + 1)
    d, h, w = D // 2, H // 2, W // 2
    x = torch.randn(N, d, h, w, c)
    xa, xu = _pair(x, (N, d, h, w, c), torch.bfloat16)
    oa = torch.empty(N, D, H, W, c, dtype=torch.bfloat16, device="cuda")
    ou = torch.zeros((oa.numel() + 1,), dtype=torch.bfloat16, device="cuda")[1:].view(oa.shape)
    assert L.lbm_nn_upsample2(_p(xa), _p(oa), N, d, h, w, c, _s()) == 0
    assert L.lbm_nn_upsample2(_p(xu), _p(ou), N, d, h, w, c, _s()) == 0
    _same(oa, ou)
    g = torch.randn(N, D, H, W, c)
    ga, gu = _pair(g, (N, D, H, W, c), torch.bfloat16)
    m = torch.randn(N, d, h, w, c)
    ma, mu = _pair(m, (N, d, h, w, c), torch.bfloat16)
    ia = torch.empty(N, d, h, w, c, dtype=torch.bfloat16, device="cuda")
    iu = torch.zeros((ia.numel() + 1,), dtype=torch.bfloat16, device="cuda")[1:].view(ia.shape)
    assert L.lbm_nn_upsample2_bwd(_p(ga), _p(ia), _p(ma), N, d, h, w, c, _s()) == 0
    assert L.lbm_nn_upsample2_bwd(_p(gu), _p(iu), _p(mu), N, d, h, w, c, _s()) == 0
    _same(ia, iu)


@pytest.mark.parametrize("ca,cb", [(32, 16), (64, 32)])
def test_concat_and_split_vector_equals_elementwise(ca, cb):
    import torch
    L = _lib()
    torch.manual_seed(ca + cb)
    nv = N * D * H * W
    a = torch.randn(nv, ca)
    b = torch.randn(nv, cb)
    aa, au = _pair(a, (nv, ca), torch.bfloat16)
    ba, bu = _pair(b, (nv, cb), torch.bfloat16)
    oa = torch.empty(nv, ca + cb, dtype=torch.bfloat16, device="cuda")
    ou = torch.zeros((oa.numel() + 1,), dtype=torch.bfloat16, device="cuda")[1:].view(oa.shape)
    assert L.lbm_nn_concat(_p(aa), ca, _p(ba), cb, _p(oa), nv, _s()) == 0
    assert L.lbm_nn_concat(_p(au), ca, _p(bu), cb, _p(ou), nv, _s()) == 0
    _same(oa, ou)
    torch.cuda.synchronize()
    assert torch.equal(oa[:, :ca], aa) and torch.equal(oa[:, ca:], ba)
    g = torch.randn(nv, ca + cb)
    gA, gU = _pair(g, (nv, ca + cb), torch.bfloat16)
    m = torch.randn(nv, cb)
    ma, mu = _pair(m, (nv, cb), torch.bfloat16)
    prev = torch.randn(nv, cb)
    for acc in (0, 1):
        xa = torch.empty(nv, ca, dtype=torch.bfloat16, device="cuda")
        xu = torch.zeros((xa.numel() + 1,), dtype=torch.bfloat16, device="cuda")[1:].view(xa.shape)
        ya, yu = _pair(prev, (nv, cb), torch.bfloat16)
        assert L.lbm_nn_split(_p(gA), ca, cb, _p(xa), _p(ya), _p(ma), acc, nv, _s()) == 0
        assert L.lbm_nn_split(_p(gU), ca, cb, _p(xu), _p(yu), _p(mu), acc, nv, _s()) == 0
        _same(xa, xu)
        _same(ya, yu)


def test_head_weight_gradient_one_pass_matches_fp64_and_general_form():
    import torch
    L = _lib()
    torch.manual_seed(7)
    nv, cin, cout = 50_000, 16, 4
    gy = torch.randn(nv, cout, device="cuda")
    w = torch.randn(cout, cin, device="cuda")
    x = torch.randn(nv, cin)
    xa, xu = _pair(x, (nv, cin), torch.bfloat16)
    scr = torch.empty(256 * (cout * cin + cout), device="cuda")
    gx = torch.empty(nv, cin, dtype=torch.bfloat16, device="cuda")
    out = []
    for xx in (xa, xu):
        dwdb = torch.empty(cout * cin + cout, device="cuda")
        assert L.lbm_nn_head_bwd_act(_p(gy), _p(w), _p(xx), None, _p(gx), _p(dwdb), _p(scr), nv, cin, cout, 0,
                                     _s()) == 0
        torch.cuda.synchronize()
        out.append(dwdb.cpu().numpy().astype(np.float64))
    g64 = gy.cpu().numpy().astype(np.float64)
    x64 = xa.float().cpu().numpy().astype(np.float64)
    ref = np.concatenate([(g64.T @ x64).reshape(-1), g64.sum(axis=0)])
    for o in out:
        assert np.abs(o - ref).max() / np.abs(ref).max() < 1e-5
    assert np.abs(out[0] - out[1]).max() / np.abs(ref).max() < 1e-5


@pytest.mark.parametrize("nvox", [1, 255, 256, 257, 4801])
@pytest.mark.parametrize("act", [0, 1])
def test_head_vector_equals_elementwise(nvox, act):
    """The 16 -> 4 head, forward and backward data: aligned tensors (whole vectors) against shifted ones."""
    import torch
    L = _lib()
    torch.manual_seed(nvox)
    x = torch.randn(nvox, 16)
    xa, xu = _pair(x if act else x.relu(), (nvox, 16), torch.bfloat16)
    w, b = torch.randn(4, 16).cuda(), torch.randn(4).cuda()
    ya, yu = _pair(torch.zeros(nvox, 4), (nvox, 4), torch.float32)
    assert L.lbm_nn_head(_p(xa), _p(w), _p(b), _p(ya), nvox, 16, 4, _s()) == 0
    assert L.lbm_nn_head(_p(xu), _p(w), _p(b), _p(yu), nvox, 16, 4, _s()) == 0
    _same(ya, yu)
    gy = torch.randn(nvox, 4).cuda()
    ga, gu = _pair(torch.zeros(nvox, 16), (nvox, 16), torch.bfloat16)
    scr, dwdb = torch.empty(256 * 68, device="cuda"), torch.empty(68, device="cuda")
    for xx, gx in ((xa, ga), (xu, gu)):
        assert L.lbm_nn_head_bwd_act(_p(gy), _p(w), _p(xx), _p(xx), _p(gx), _p(dwdb), _p(scr), nvox, 16, 4, act,
                                     _s()) == 0
    _same(ga, gu)


def test_adam_many_equals_single_tensor_steps_and_refresh():
    import torch
    from taichi_lbm3d_gb300.unet import UNet3D
    L = _lib()
    m = UNet3D(seed=3)
    g = torch.Generator(device="cuda").manual_seed(1)
    for t in list(m.gw.values()) + list(m.gb.values()) + [m.ghw_hb]:
        t.copy_(torch.randn(t.shape, generator=g, device="cuda") * 1e-2)
    params = [(k, p, q) for k, p, q in [(k, m.w[k], m.gw[k]) for k in m.w] + [(None, m.b[k], m.gb[k]) for k in m.b]
              + [(None, m.hw, m.ghw_hb[:64].view(4, 16)), (None, m.hb, m.ghw_hb[64:])]]
    ref = [(p.clone(), torch.zeros_like(p), torch.zeros_like(p)) for _, p, _ in params]
    for step in (1, 2, 3):
        m.adam_step(lr=1e-3, weight_decay=1e-2)
        for (_, _, q), (p, mm, vv) in zip(params, ref):
            assert L.lbm_nn_adam(_p(p), _p(q), _p(mm), _p(vv), None, p.numel(), 1e-3, 0.9, 0.999, 1e-8, step, 1e-2,
                                 _s()) == 0
    for (_, p, _), (r, _, _) in zip(params, ref):
        _same(p, r)
    w16, wt16 = {k: v.clone() for k, v in m.w16.items()}, {k: v.clone() for k, v in m.wt16.items()}
    m.refresh()
    for k in m.w16:
        _same(w16[k], m.w16[k])
        _same(wt16[k], m.wt16[k])


@pytest.mark.parametrize("c,cs,dims", [(32, 16, (2, 3, 4, 5)), (64, 32, (1, 1, 1, 1)), (8, 24, (1, 2, 5, 3))])
def test_upcat_equals_upsample_then_concat(c, cs, dims):
    import torch
    L = _lib()
    torch.manual_seed(c)
    n, d, h, w = dims
    big = (n, 2 * d, 2 * h, 2 * w)
    nv = int(np.prod(big))
    bf = dict(dtype=torch.bfloat16, device="cuda")
    low, skip = torch.randn(n, d, h, w, c).cuda().to(torch.bfloat16), torch.randn(*big, cs).cuda().to(torch.bfloat16)
    up, cat, one = torch.empty(*big, c, **bf), torch.empty(*big, c + cs, **bf), torch.zeros(*big, c + cs, **bf)
    assert L.lbm_nn_upsample2(_p(low), _p(up), n, d, h, w, c, _s()) == 0
    assert L.lbm_nn_concat(_p(up), c, _p(skip), cs, _p(cat), nv, _s()) == 0
    assert L.lbm_nn_upcat(_p(low), c, _p(skip), cs, _p(one), n, d, h, w, _s()) == 0
    _same(cat, one)
    g = torch.randn(*big, c + cs).cuda().to(torch.bfloat16)
    for mask in (None, low):
        gu, gs, gl = torch.empty(*big, c, **bf), torch.empty(*big, cs, **bf), torch.empty(n, d, h, w, c, **bf)
        gl1, gs1 = torch.zeros_like(gl), torch.zeros_like(gs)
        assert L.lbm_nn_split(_p(g), c, cs, _p(gu), _p(gs), None, 0, nv, _s()) == 0
        assert L.lbm_nn_upsample2_bwd(_p(gu), _p(gl), _p(mask), n, d, h, w, c, _s()) == 0
        assert L.lbm_nn_upcat_bwd(_p(g), c, cs, _p(gl1), _p(mask), _p(gs1), n, d, h, w, _s()) == 0
        _same(gl, gl1)
        _same(gs, gs1)
    assert L.lbm_nn_upcat(_p(low), 12, _p(skip), cs, _p(one), n, d, h, w, _s()) != 0

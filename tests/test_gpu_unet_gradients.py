"""Adam takes gradient tensors of any strides, as a program that fills them in itself may hold."""
import pytest

pytestmark = pytest.mark.gpu


def test_adam_step_with_strided_gradients():
    import torch
    from taichi_lbm3d_gb300.unet import UNet3D
    runs = []
    for strided in (False, True):
        m = UNet3D(seed=3)
        g = torch.Generator(device="cuda").manual_seed(1)
        for t in list(m.gw.values()) + list(m.gb.values()) + [m.ghw_hb]:
            t.copy_(torch.randn(t.shape, generator=g, device="cuda") * 1e-2)
        if strided:
            for k in m.gw:
                m.gw[k] = m.gw[k].transpose(0, 2).contiguous().transpose(0, 2)
            for k in m.gb:
                m.gb[k] = torch.stack([m.gb[k], m.gb[k] + 1], 1)[:, 0]
            m.ghw_hb = torch.stack([m.ghw_hb, m.ghw_hb - 1], 1)[:, 0].contiguous()
        for _ in range(2):
            m.adam_step(lr=1e-3, weight_decay=1e-2)
        runs.append({**{"w_" + k: v for k, v in m.w.items()}, **{"b_" + k: v for k, v in m.b.items()}, "hw": m.hw,
                     "hb": m.hb, **{"w16_" + k: v for k, v in m.w16.items()}})
    for k, v in runs[0].items():
        assert torch.equal(v, runs[1][k]), k

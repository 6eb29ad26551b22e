"""Bias gradients for every way that channels divide a block (whole pixels of eight
channels a thread, of any number of channels, more channels than threads), and weight
gradients on image rows shorter than the 16 pixels between a thread's copies."""
import pytest

from test_unet_tiles_gpu import F32_TOL, bf, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [1, 2, 3, 4, 7, 12, 16, 20, 40, 56, 64, 96, 128, 184, 255, 256, 257, 264, 300, 520, 1000, 2048, 2056])
@pytest.mark.parametrize("shift", [0, 1])
def test_bias_gradient(C, shift):
    import torch

    from kwave_gb300 import unet_ops as U

    for npix in (1, 3, 1030, 5000):
        dz = bf((npix * C + shift,), C + npix)
        db = torch.ones(C, dtype=torch.float32, device="cuda")
        U.bias_grad(dz.cuda()[shift:].reshape(npix, C), db)
        ref = dz[shift:].double().reshape(npix, C)
        e = (db.cpu().double() - 1 - ref.sum(0)).abs() / (1 + ref.abs().sum(0))
        assert float(e.max()) <= F32_TOL, npix


@pytest.mark.parametrize("nb,H,W,c1,c2,cout", [(3, 7, 1, 8, 0, 8), (2, 6, 2, 16, 8, 16), (5, 4, 10, 8, 16, 24), (2, 9, 15, 40, 0, 32),
                                               (1, 10, 16, 16, 0, 40), (2, 4, 18, 24, 32, 8)])
def test_weight_gradient_of_short_rows(nb, H, W, c1, c2, cout):
    import torch
    import torch.nn.functional as F

    from kwave_gb300 import unet_ops as U

    x1, dz = bf((nb, H, W, c1), 1), bf((nb, H, W, cout), 2)
    x2 = bf((nb, H // 2, W // 2, c2), 3) if c2 else None
    dw = torch.zeros((cout, 9, c1 + c2), dtype=torch.float32, device="cuda")
    U.conv3x3_wgrad(x1.cuda(), dz.cuda(), dw, x2=x2.cuda() if c2 else None)
    x = x1.float().permute(0, 3, 1, 2)
    if c2:
        x = torch.cat([x, F.interpolate(x2.float().permute(0, 3, 1, 2), scale_factor=2, mode="nearest")], dim=1)
    wt = torch.zeros((cout, c1 + c2, 3, 3), requires_grad=True)
    F.conv2d(x, wt, None, padding=1).backward(dz.float().permute(0, 3, 1, 2))
    assert rel(dw.reshape(cout, 3, 3, c1 + c2).permute(0, 3, 1, 2), wt.grad) <= F32_TOL

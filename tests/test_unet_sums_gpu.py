"""Bias gradients for every way that channels divide a block (whole pixels of eight
channels a thread, of any number of channels, more channels than threads)."""
import pytest

from test_unet_tiles_gpu import F32_TOL, bf

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

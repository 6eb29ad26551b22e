"""The gathered tensor-core tiles of the U-Net convolutions (k_umma) at the edges
of their dispatch, against torch in float32 on the same bf16 values: image widths
that are and are not multiples of the 64-pixel chunk, odd widths, one tile and
many, the upsampled concatenation, tile widths from 16 to 256 columns with ragged
last tiles, and sums split over CTAs.  Tolerance: 1e-5 relative L2, float32
accumulation of up to 13 k products against float32 references."""
import pytest

pytestmark = pytest.mark.gpu

F32_TOL = 1e-5


def rel(a, b):
    a, b = a.detach().double().cpu(), b.detach().double().cpu()
    return float((a - b).norm() / max(float(b.norm()), 1e-300))


def bf(shape, seed, scale=1.0):
    import torch

    return (scale * torch.randn(shape, generator=torch.Generator().manual_seed(seed))).to(torch.bfloat16)


@pytest.mark.parametrize("nb,H,W,c1,c2,cout", [
    (1, 5, 7, 8, 0, 8),        # less than one tile
    (3, 9, 24, 24, 0, 72),     # a ragged tile in every dimension
    (2, 16, 64, 32, 16, 192),  # one image row per chunk, concatenation, 192 columns
    (1, 12, 192, 16, 0, 16),   # three chunks per row
    (2, 6, 40, 40, 24, 256),   # chunks across rows and images, concatenation
    (1, 32, 32, 256, 0, 256),  # K split over CTAs
    (4, 40, 40, 128, 0, 128),
    (2, 64, 64, 96, 160, 144),
    (1, 4, 128, 64, 128, 192),  # rows of 128 pixels, too wide an output for the halo tiles
])
def test_gathered_tiles(nb, H, W, c1, c2, cout):
    import torch
    import torch.nn.functional as F

    from kwave_gb300 import unet_ops as U

    x1, dz = bf((nb, H, W, c1), 1), bf((nb, H, W, cout), 2)
    x2 = bf((nb, H // 2, W // 2, c2), 3) if c2 else None
    w = bf((cout, 9, c1 + c2), 4, 0.1)
    bias = torch.randn(cout, generator=torch.Generator().manual_seed(5))
    x2d = x2.cuda() if c2 else None
    _, yf = U.conv3x3(x1.cuda(), w.cuda(), bias.cuda(), relu=True, x2=x2d,
                      yf=torch.empty((nb, H, W, cout), dtype=torch.float32, device="cuda"))
    dw = torch.zeros((cout, 9, c1 + c2), dtype=torch.float32, device="cuda")
    U.conv3x3_wgrad(x1.cuda(), dz.cuda(), dw, x2=x2d)
    torch.cuda.synchronize()

    x = x1.float().permute(0, 3, 1, 2)
    if c2:
        x = torch.cat([x, F.interpolate(x2.float().permute(0, 3, 1, 2), scale_factor=2, mode="nearest")], dim=1)
    wt = w.float().reshape(cout, 3, 3, c1 + c2).permute(0, 3, 1, 2).requires_grad_(True)
    y = F.conv2d(x, wt, None, padding=1)
    y.backward(dz.float().permute(0, 3, 1, 2))
    e_y = rel(yf, torch.relu(y + bias[:, None, None]).permute(0, 2, 3, 1))
    e_w = rel(dw.reshape(cout, 3, 3, c1 + c2).permute(0, 3, 1, 2), wt.grad)
    print(f"{nb}x{H}x{W} {c1}+{c2}->{cout}: forward {e_y:.2e} weight gradient {e_w:.2e}")
    assert e_y <= F32_TOL and e_w <= F32_TOL


@pytest.mark.parametrize("npix,C", [(1, 8), (77, 24), (1000, 32), (4097, 48), (70000, 8), (513, 2048), (5, 4104)])
@pytest.mark.parametrize("shift", [0, 1])  # 1: tensors that do not start on 16 bytes
def test_elementwise_gradients(npix, C, shift):
    """ReLU and bias gradients, eight values per access and one by one."""
    import torch

    from kwave_gb300 import unet_ops as U

    n = npix * C
    dy, y = bf((n + shift,), 6), bf((n + shift,), 7)
    y[shift::3] = 0.0
    dz = U.relu_grad(dy.cuda()[shift:], y.cuda()[shift:])
    db = torch.ones(C, dtype=torch.float32, device="cuda")
    U.bias_grad(dy.cuda()[shift:].reshape(npix, C), db)
    torch.cuda.synchronize()
    assert torch.equal(dz.cpu(), torch.where(y[shift:].float() > 0, dy[shift:], torch.zeros_like(dy[shift:])))
    ref = dy[shift:].double().reshape(npix, C)
    e = float((db.cpu().double() - 1 - ref.sum(0)).norm() / (1 + ref.abs().sum(0)).norm())
    assert e <= F32_TOL


@pytest.mark.parametrize("cout,cin", [(8, 8), (32, 32), (40, 72), (256, 8)])
def test_flipped_weights(cout, cin):
    import torch

    from kwave_gb300 import unet_ops as U

    w = bf((cout, 9, cin), 8)
    assert torch.equal(U.flip_weights(w.cuda()).cpu(), w.flip(1).permute(2, 1, 0).contiguous())

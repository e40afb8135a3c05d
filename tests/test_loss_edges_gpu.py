"""GPU edge cases of the strip-walking L1 + D-SSIM kernel: widths around its 118-column strips, heights
around its 16-row chunks, windows wider than the image, a skipped bottom, and a gradient that is written
over one of the images.  The oracle is the reference formulation in PyTorch FP32 (conv2d and autograd);
loss within 1e-5 relative, gradient within 1e-3 normwise (the separable window rounds differently)."""
import pytest
import torch

from omnigs_b200 import train
from test_train_gpu import _rel, ref_l1_dssim

pytestmark = pytest.mark.gpu


def _images(H, W):
    gen = torch.Generator(device="cpu").manual_seed(H * 4099 + W)
    gt = torch.rand(3, H, W, generator=gen).cuda()
    return (gt + 0.1 * torch.randn(3, H, W, generator=gen).cuda()).clamp(0, 1), gt


@pytest.mark.parametrize("H,W,rows", [(1, 1, 1), (3, 7, 2), (16, 118, 16), (17, 119, 17), (15, 117, 15), (33, 236, 32),
                                      (40, 237, 23), (700, 33, 700), (129, 1000, 128)])
def test_l1_dssim_edges(cuda, H, W, rows):
    img, gt = _images(H, W)
    loss, grad = train.l1_dssim(img, gt, 0.2, rows=rows)
    x = img.clone().requires_grad_(True)
    ref = ref_l1_dssim(x, gt, 0.2, rows)
    ref[0].backward()
    for got, want in zip(loss.tolist(), ref):
        assert abs(got - want.item()) <= 1e-5 * abs(want.item())
    assert _rel(grad, x.grad) < 1e-3
    assert rows == H or grad[:, rows:].abs().max().item() == 0.0


@pytest.mark.parametrize("over", ["img", "gt"])
def test_l1_dssim_gradient_over_an_image(cuda, over):
    img, gt = _images(50, 130)
    loss, grad = train.l1_dssim(img, gt, 0.2)
    out = img if over == "img" else gt
    loss2, grad2 = train.l1_dssim(img, gt, 0.2, dL_dimage=out)
    assert torch.equal(loss, loss2) and torch.equal(grad, grad2) and grad2.data_ptr() == out.data_ptr()

"""GPU tests of the loss on small, tall and narrow images, and of the Adam step with gradients that start anywhere (slices
of one flat buffer): results, and that such gradients cost little more than aligned ones."""
import pytest
import torch

from omnigs_b200 import train

pytestmark = pytest.mark.gpu


def _reference(img, gt, rows, lam=0.2):
    """(loss, l1, ssim) and dL/dimg in float64 (11-tap Gaussian window of sigma 1.5, zero padding)."""
    a = img.double().requires_grad_(True)
    C = img.shape[0]
    w = torch.exp(-(torch.arange(11, dtype=torch.float64, device=img.device) - 5) ** 2 / (2 * 1.5 ** 2))
    w = w / w.sum()

    def blur(v):
        v = torch.nn.functional.conv2d(v, w.view(1, 1, 1, 11).expand(C, 1, 1, 11), padding=(0, 5), groups=C)
        return torch.nn.functional.conv2d(v, w.view(1, 1, 11, 1).expand(C, 1, 11, 1), padding=(5, 0), groups=C)

    x, y = a[None, :, :rows], gt.double()[None, :, :rows]
    m1, m2 = blur(x), blur(y)
    s1, s2, s12 = blur(x * x) - m1 * m1, blur(y * y) - m2 * m2, blur(x * y) - m1 * m2
    ssim = (((2 * m1 * m2 + 1e-4) * (2 * s12 + 9e-4)) / ((m1 * m1 + m2 * m2 + 1e-4) * (s1 + s2 + 9e-4))).mean()
    l1 = (x - y).abs().mean()
    loss = (1 - lam) * l1 + lam * (1 - ssim)
    return torch.stack([loss, l1, ssim]).detach(), torch.autograd.grad(loss, a)[0]


@pytest.mark.parametrize("C,H,W,rows", [(3, 1, 1, 1), (1, 5, 3, 5), (3, 16, 16, 16), (3, 16, 16, 7), (2, 4, 118, 4), (3, 9, 119, 9),
                                        (1, 17, 237, 13), (3, 700, 16, 700), (3, 333, 27, 300), (5, 64, 91, 64), (3, 40, 700, 40)])
@pytest.mark.parametrize("in_place", [False, True])
def test_loss_of_small_images(cuda, C, H, W, rows, in_place):
    g = torch.Generator(device=cuda).manual_seed(H * 1000 + W)
    gt = torch.rand(C, H, W, generator=g, device=cuda)
    img = (gt + 0.1 * torch.randn(C, H, W, generator=g, device=cuda)).clamp_min(0)
    ref, dref = _reference(img, gt, rows)
    d = img if in_place else torch.full_like(img, 7.0)
    loss, d = train.l1_dssim(img, gt, 0.2, rows=rows, dL_dimage=d, loss=torch.empty(3, device=cuda),
                             workspace=train.l1_dssim_workspace(C, H, W))
    torch.cuda.synchronize()
    assert (loss.double() - ref).abs().max() < 1e-5
    assert (d.double() - dref).abs().max() < 1e-3 * dref.abs().max()
    assert bool((d[:, rows:] == 0).all())


def _us(f, n=30):
    for _ in range(3):
        f()
    best = float("inf")
    for _ in range(8):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(n):
            f()
        b.record()
        torch.cuda.synchronize()
        best = min(best, 1000 * a.elapsed_time(b) / n)
    return best


def _adam(P, M, offset):
    g = torch.Generator(device="cuda").manual_seed(P + M)
    n = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    raw = [2 * n(P, 3), n(P, 1, 3), 0.1 * n(P, M - 1, 3), n(P, 1), 0.5 * n(P, 3) - 4, n(P, 4)]
    grads = [1e-4 * n(P, 3), 1e-4 * n(P, M, 3), 1e-4 * n(P, 1), 1e-3 * n(P, 3), 1e-4 * n(P, 4)]
    flat = torch.cat([torch.zeros(offset, device="cuda")] + [t.reshape(-1) for t in grads])
    out, at = [], offset
    for t in grads:
        out.append(flat[at:at + t.numel()].view(t.shape))
        at += t.numel()
    return train.GaussianModelState(*raw), out


@pytest.mark.parametrize("P,M", [(1, 1), (7, 4), (255, 16), (257, 16), (1023, 9), (1537, 1), (5001, 16)])
def test_adam_from_one_flat_buffer(cuda, P, M):
    got = []
    for offset in (0, 1, 3):
        model, grads = _adam(P, M, offset)
        for _ in range(3):
            model.adam_step(*grads)
        torch.cuda.synchronize()
        got.append([t.clone() for t in (*model.params, *model.m, *model.v, model.shs, model.scales)])
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))


def test_unaligned_gradients_cost_little_more(cuda):
    def t(offset):
        model, grads = _adam(100000, 16, offset)
        return _us(lambda: model.adam_step(*grads))

    # (the same loads one float at a time: 64 us against 42 before they were in flight together)
    assert t(1) < 1.4 * t(0)

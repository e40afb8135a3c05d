"""GPU edge cases of the fused Adam step, which updates the SH coefficients in tiles of 32 Gaussians and
the other groups in chunks of 1536 values with 16-byte accesses: sizes around both, every SH count that
changes the row length's alignment, BF16 SH, and gradients that do not start on 16 bytes.  The oracle is
the reference's Adam and activations in PyTorch FP64 over two steps; values within 1e-5 of the largest
(FP32 arithmetic of torch's own formula order), BF16 SH within one rounding of that."""
import math

import pytest
import torch

from omnigs_b200 import train

pytestmark = pytest.mark.gpu


def _off(t):
    """The same values at an address that is 4 bytes past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 4, device=t.device)
    out = buf[1:1 + t.numel()].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 16 == 4
    return out


@pytest.mark.parametrize("P,M,bf16,aligned", [
    (1, 16, False, True), (31, 16, False, True), (32, 16, True, True), (33, 16, False, True), (512, 1, False, True),
    (513, 4, True, True), (1537, 9, False, True), (3000, 2, False, True), (1000, 16, False, False),
    (70, 3, True, False)])
def test_adam_step_edges(cuda, P, M, bf16, aligned):
    gen = torch.Generator(device="cpu").manual_seed(P * 31 + M)
    r = lambda *s: torch.randn(*s, generator=gen).cuda()  # noqa: E731
    raw = [r(P, 3), r(P, 1, 3), 0.1 * r(P, M - 1, 3), r(P, 1), math.log(0.02) + 0.5 * r(P, 3), r(P, 4)]
    model = train.GaussianModelState(*raw, sh_bf16=bf16)
    p = [t.double() for t in raw]
    m, v = [torch.zeros_like(t) for t in p], [torch.zeros_like(t) for t in p]
    lr = [model.lr[k] for k in train.GROUPS]
    for step in (1, 2):
        grads = [r(P, 3), r(P, M, 3), r(P, 1), r(P, 3), r(P, 4)]
        model.adam_step(*(grads if aligned else [_off(g) for g in grads]))
        dx, dsh, do, ds, dq = (g.double() for g in grads)
        o, e, n = torch.sigmoid(p[3]), torch.exp(p[4]), p[5].norm(dim=1, keepdim=True)
        y = p[5] / n
        g = [dx, dsh[:, :1], dsh[:, 1:], do * o * (1 - o), ds * e, (dq - y * (y * dq).sum(1, keepdim=True)) / n]
        for i in range(6):
            m[i] = 0.9 * m[i] + 0.1 * g[i]
            v[i] = 0.999 * v[i] + 0.001 * g[i] * g[i]
            p[i] = p[i] - lr[i] / (1 - 0.9 ** step) * m[i] / ((v[i] / (1 - 0.999 ** step)).sqrt() + 1e-15)
    close = lambda a, b, tol=1e-5: a.numel() == 0 or \
        float((a.double() - b).abs().max()) <= tol * float(b.abs().max())  # noqa: E731
    for i in range(6):
        assert close(model.params[i], p[i]) and close(model.m[i], m[i]) and close(model.v[i], v[i]), train.GROUPS[i]
    assert close(model.shs, torch.cat([p[1], p[2]], 1), 2.0 ** -8 if bf16 else 1e-5)
    assert close(model.opacities, torch.sigmoid(p[3])) and close(model.scales, torch.exp(p[4]))
    assert close(model.rotations, p[5] / p[5].norm(dim=1, keepdim=True))

"""GPU test of what the backward blend does to pixels that a splat does not reach: nothing, exactly.  Their transmittance is
multiplied by the approximate reciprocal of 1 for every candidate of the warp, which has to be 1, or hundreds of splats
elsewhere in an 8x8 patch would move a pixel's gradients."""
import numpy as np
import pytest
import torch

from omnigs_b200 import lonlat, scenes

pytestmark = pytest.mark.gpu

W, H = 256, 128


def _at(px, py, r):
    """The point at distance r that projects to pixel (px, py) of the identity view."""
    lon, lat = np.pi * ((2 * px + 1) / W - 1), 0.5 * np.pi * ((2 * py + 1) / H - 1)
    return r * np.array([np.sin(lon) * np.cos(lat), np.sin(lat), np.cos(lon) * np.cos(lat)])


def _gradients(means, opacities):
    P = len(means)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()  # noqa: E731
    rng = np.random.default_rng(0)
    g = lonlat.GaussianTensors(t(means), t(opacities).view(P, 1), colors_precomp=t(rng.random((P, 3))),
                               cov3D_precomp=t(np.tile([1e-8, 0, 0, 1e-8, 0, 1e-8], (P, 1))))
    cam = lonlat.Camera.from_view(scenes.make_view(W, H, (0.0, 0.0, 0.0), np.eye(3)), background=(0.2, 0.4, 0.6))
    _, radii, n, state = lonlat.rasterize(g, cam)
    grads = lonlat.Gradients.empty(P, 0, "cuda")
    state.backward(g, cam, radii, torch.from_numpy(scenes.upstream_grad(W, H, seed=1)).cuda(), grads, R=n)
    torch.cuda.synchronize()
    return torch.cat([grads.dL_dopacity, grads.dL_dcolors, grads.dL_dmeans3D, grads.dL_dcov3D], 1)


@pytest.mark.parametrize("others", [1, 100, 700])
def test_gradients_ignore_splats_elsewhere_in_the_patch(cuda, others):
    # patch of columns 128-135 and rows 64-71: one splat around (130, 66), the others behind it around (134, 70), each
    # within 1.9 pixels (0.3 of dilation alone)
    rng = np.random.default_rng(others)
    one = _at(130.2, 66.1, 1.0)[None]
    rest = np.stack([_at(134.0 + 0.2 * a, 70.0 + 0.2 * b, 2.0 + 0.001 * k)
                     for k, (a, b) in enumerate(rng.random((others, 2)))])
    alone = _gradients(one, np.array([0.9]))
    both = _gradients(np.concatenate([one, rest]), np.concatenate([[0.9], np.full(others, 0.02)]))
    assert float(alone.abs().max()) > 0 and float(both[1:].abs().max()) > 0
    assert torch.equal(alone[0], both[0])

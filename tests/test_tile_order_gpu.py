"""GPU test of the blends' tile order: above a number of Gaussians the blends take the tiles heaviest first,
below it in order.  The same visible Gaussians are rendered both ways, the second time padded with Gaussians
inside the near-cull sphere, at sizes with one tile, a partial segment of tiles and more than one segment:
image, radii and per-pixel state equal bit for bit (the output is filled with NaN before), gradients to the
run-to-run variation of the blend's float atomics (1e-5 normwise)."""
import numpy as np
import pytest
import torch

import helpers
from omnigs_b200 import batch, lonlat, scenes

pytestmark = pytest.mark.gpu

GRADS = ("dL_dopacity", "dL_dmeans3D", "dL_dscales", "dL_drotations", "dL_dsh")


def _scenes(P, padded):
    g = scenes.make_gaussians(padded, seed=padded, pole_fraction=0.4)
    m = g.means3D[P:]
    m *= np.float32(0.15) / np.linalg.norm(m, axis=1, keepdims=True)
    few = scenes.Gaussians(g.means3D[:P], g.scales[:P], g.rotations[:P], g.opacities[:P], g.shs[:P])
    return [lonlat.GaussianTensors.from_numpy(x) for x in (few, g)]


@pytest.mark.parametrize("P,padded,W,H", [(500, 262144, 16, 16), (9000, 262144, 300, 130), (12000, 300000, 2080, 1040)])
def test_tile_order(cuda, P, padded, W, H):
    cam = lonlat.Camera.from_view(scenes.identity_view(W, H), background=(0.1, 0.2, 0.3))
    dpix = torch.from_numpy(scenes.upstream_grad(W, H, seed=3)).cuda()
    runs = []
    for gt in _scenes(P, padded):
        _, _, n, _ = lonlat.rasterize(gt, cam)
        state = lonlat.LonlatState(gt.P, W, H, n + 64)
        out = torch.full((3, H, W), float("nan"), device=cuda)
        radii = torch.empty(gt.P, dtype=torch.int32, device=cuda)
        state.forward(gt, cam, out, radii)
        grads = lonlat.Gradients.empty(gt.P, gt.M, cuda)
        state.backward(gt, cam, radii, dpix, grads)
        torch.cuda.synchronize()
        iv = state.image_view()
        runs.append((out, radii[:P], iv["final_T"].clone(), iv["n_contrib"].clone(), iv["ranges"].clone(), grads))
    for x, y in zip(runs[0][:5], runs[1][:5]):
        assert torch.equal(x, y)
    for name in GRADS:
        a, b = (helpers.to_np(getattr(r[5], name)) for r in runs)
        assert helpers.normwise_rel(b[:P], a) < 1e-5, name
        assert not b[P:].any(), name


def test_tile_order_batch(cuda):
    # (all cameras at the origin, where the padding is culled)
    views = [scenes.make_view(W, H, (0.0, 0.0, 0.0), scenes.rotation_yaw_pitch(0.5 * k, 0.2 * k))
             for k, (W, H) in enumerate([(500, 250), (33, 17), (1024, 512), (130, 40)])]
    cams = batch.BatchCameras.from_views(views)
    dl = [torch.from_numpy(scenes.upstream_grad(W, H, seed=W)).cuda() for W, H in cams.sizes]
    runs = []
    for gt in _scenes(7000, 70000):
        images, _, state = batch.render_batch(gt, cams)
        grads = batch.BatchGradients.empty(gt.P, gt.M, cuda)
        state.backward(gt, cams, dl, grads)
        torch.cuda.synchronize()
        runs.append((images, grads))
    for x, y in zip(runs[0][0], runs[1][0]):
        assert torch.equal(x, y)
    for name in GRADS:
        a, b = (helpers.to_np(getattr(r[1], name)) for r in runs)
        assert helpers.normwise_rel(b[:7000], a) < 1e-5, name

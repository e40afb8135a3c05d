"""GPU edge cases of the tile blends: images that are not whole tiles, one-pixel images, lists longer than
every staging batch, and splats on either side of the rule that leaves the 0.99 clamp and the exponent's
sign test out (opacities around and above the clamp, among them 0 and 1), at every batch size, with the
per-pixel state stored and recomputed.

Tolerances: gradients <= 1e-3 normwise; image <= 1e-4, except at pixels where FP32 and FP64 decide
alpha >= 1/255 differently (relative rounding ~1e-6 of a decision spread over several decades: under one
pixel in a thousand), which may be off by one splat's 1/255 times its colour."""
import numpy as np
import pytest
import torch

import helpers
from omnigs_b200 import batch, lonlat, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("staged", [128, 256, 512])
@pytest.mark.parametrize("P,W,H,grow", [(1, 1, 1, 1.0), (40, 17, 9, 20.0), (3000, 100, 50, 3.0), (6000, 33, 31, 1.0),
                                        (4000, 250, 120, 0.3)])
def test_blend_edges(cuda, P, W, H, grow, staged):
    g = scenes.make_gaussians(P, seed=P, pole_fraction=0.05)
    rng = np.random.default_rng(P)
    special = rng.random((P, 1)) < 0.3
    g.opacities[special] = rng.choice(np.float32([0.0, 0.003, 0.98, 0.98999, 0.99, 0.995, 1.0]), int(special.sum()))
    g.opacities[: P // 2][~special[: P // 2]] *= np.float32(0.05)  # long lists before saturation
    g.scales *= np.float32(grow)
    v = scenes.make_view(W, H, (0.1, 0.0, -0.2), scenes.rotation_yaw_pitch(0.4, -0.2))
    bg = (0.3, 0.2, 0.1)
    gt, cam = lonlat.GaussianTensors.from_numpy(g), lonlat.Camera.from_view(v, background=bg)
    dpix = scenes.upstream_grad(W, H, seed=P)
    try:
        batch.set_blend_batch(staged, staged)
        cu = helpers.run_cuda(gt, cam, torch.from_numpy(dpix).cuda())
        state = lonlat.LonlatState(P, W, H, cu["num_rendered"] + 16, recompute_T=True)
        out, radii = torch.empty(3, H, W, device=cuda), torch.empty(P, dtype=torch.int32, device=cuda)
        state.forward(gt, cam, out, radii)
        again = lonlat.Gradients.empty(P, gt.M, cuda)
        state.backward(gt, cam, radii, torch.from_numpy(dpix).cuda(), again)
        torch.cuda.synchronize()
    finally:
        batch.set_blend_batch(128, 128)  # the library's defaults
    assert torch.equal(out, cu["image"])
    o = helpers.oracle_stagewise(cu, g, v, dpix, np.asarray(bg, np.float32))
    err = np.abs(helpers.to_np(cu["image"]) - o["forward"]["image"]).max(0)
    assert (err > 1e-4).mean() < 1e-3
    assert err.max() < 1.0 / 255.0 * max(1.0, float(np.abs(helpers.to_np(cu["rgb"])).max())) + 1e-4
    for name, ref in (("dL_dopacity", o["render_backward"]["dL_dopacity"]), ("dL_dcolors", o["render_backward"]["dL_dcolor"]),
                      ("dL_dmeans3D", o["preprocess_backward"]["dL_dmeans3D"]), ("dL_dscales", o["preprocess_backward"]["dL_dscales"])):
        mine = helpers.to_np(getattr(cu["grads"], name))
        assert helpers.normwise_rel(mine, np.asarray(ref).reshape(mine.shape)) < 1e-3, name
        assert helpers.normwise_rel(helpers.to_np(getattr(again, name)), mine) < 1e-5, name

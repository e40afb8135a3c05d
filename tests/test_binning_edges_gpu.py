"""GPU edge cases of the binning: the counted depth order and the radix sort on either side of their
limits, images that are not whole bins of 8x4 tiles, one-tile and one-row images, splats that cover the
whole image, lists of thousands of splats per tile, more tiles than Gaussians, equal depths, and views of
uneven size with few Gaussians.  Keys, point list and ranges equal the oracle's bit for bit."""
import numpy as np
import pytest
import torch

import helpers
import oracle
from omnigs_b200 import batch, lonlat, scenes

pytestmark = pytest.mark.gpu

VIEW = ((0.2, -0.1, 0.3), scenes.rotation_yaw_pitch(0.7, 0.2))


def _check(tile_ids, point_list, ranges, W, H, radii, means2D, depths, seam=False):
    b = oracle.binning(W, H, radii, means2D, depths, None, f32=True, seam_wrap=seam)
    assert b["num_rendered"] == len(tile_ids)
    np.testing.assert_array_equal(tile_ids, (b["keys"] >> np.uint64(32)).astype(np.uint32))
    np.testing.assert_array_equal(point_list, b["point_list"])
    np.testing.assert_array_equal(ranges, b["ranges"])


@pytest.mark.parametrize("P,W,H,grow", [
    (1, 16, 16, 1.0), (3, 1, 1, 1.0), (5000, 16, 16, 1.0), (300, 17, 65, 1.0), (3000, 2048, 16, 1.0),
    (700, 40, 600, 1.0), (12288, 512, 256, 1.0), (12289, 512, 256, 1.0), (12288, 2048, 1024, 1.0),
    (40000, 1520, 712, 1.0), (2000, 500, 250, 30.0), (30000, 500, 250, 4.0), (200000, 130, 70, 1.0),
    (40, 4096, 2048, 1.0), (9000, 4096, 2048, 1.0), (20000, 2048, 1024, 1.0)])
def test_binning_edges(cuda, P, W, H, grow):
    g = scenes.make_gaussians(P, seed=P + W, pole_fraction=0.1)
    g.scales *= np.float32(grow)
    g.means3D[P // 2:] = g.means3D[:P - P // 2]  # equal depths: the index decides
    cu = helpers.run_cuda(lonlat.GaussianTensors.from_numpy(g), lonlat.Camera.from_view(scenes.make_view(W, H, *VIEW)))
    n = helpers.to_np
    _check(n(cu["tile_ids"]).view(np.uint32), n(cu["point_list"]).view(np.uint32), n(cu["ranges"]).view(np.uint32), W, H,
           n(cu["radii"]), n(cu["means2D"]), n(cu["depths"]))
    np.testing.assert_array_equal(n(cu["depth_order"]), np.argsort(n(cu["depths"]), kind="stable"))


@pytest.mark.parametrize("P,seam", [(50, False), (2000, False), (2000, True), (60000, True)])
def test_batch_binning_edges(cuda, P, seam):
    g = scenes.make_gaussians(P, seed=P, seam_fraction=0.3)
    views = scenes.random_views(5, [(500, 250), (33, 17), (1024, 512), (130, 40)], seed=P)
    cams = batch.BatchCameras.from_views(views)
    gt = lonlat.GaussianTensors.from_numpy(g)
    _, per, state = batch.render_batch(gt, cams, seam_wrap=seam)
    total = sum(per)
    sv, bv = state.state_view(), state.binning_view(total)
    torch.cuda.synchronize()
    n = helpers.to_np
    tiles, points = n(bv["tile_ids"]).view(np.uint32), n(bv["point_list"]).view(np.uint32)
    for v, (W, H) in enumerate(cams.sizes):
        base, count = sv["tile_base"][v], ((W + 15) // 16) * ((H + 15) // 16)
        mine = (tiles >= base) & (tiles < base + count)
        ranges = n(sv["ranges"][v]).view(np.uint32).astype(np.int64)
        first = ranges[ranges[:, 1] > 0, 0].min() if per[v] else 0
        ranges[ranges[:, 1] > 0] -= first
        _check(tiles[mine] - np.uint32(base), points[mine] - np.uint32(v * P), ranges.astype(np.uint32), W, H,
               n(sv["radii"][v]), n(sv["splat"][v][:, :2]), n(sv["depth"][v]), seam)
        assert mine.sum() == per[v]

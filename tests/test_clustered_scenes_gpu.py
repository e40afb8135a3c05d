"""GPU tests of the tile lists where Gaussians are not spread evenly: scenes that fall into a few bins of 8x4 tiles,
splats over the whole image, lists that end at and around a warp's piece and a block of pieces, few Gaussians under
many tiles (where the tiles' totals are kept differs), and the same in a captured graph.  Lists equal the oracle's bit
for bit.  How the Gaussians are spread changes what the lists cost by a small factor only."""
import numpy as np
import pytest
import torch

import helpers
import oracle
from omnigs_b200 import batch, capi, lonlat, scenes

pytestmark = pytest.mark.gpu


def _clustered(P, spread, grow=1.0, seed=0):
    """Gaussians whose directions lie within about `spread` radians of one (0: a shell all around)."""
    g = scenes.make_gaussians(P, seed=seed + P)
    if spread > 0:
        rng = np.random.default_rng(P)
        d = np.array([0.3, 0.1, 1.0]) + spread * rng.standard_normal((P, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        g.means3D[:] = (d * np.linalg.norm(g.means3D, axis=1, keepdims=True)).astype(np.float32)
    g.scales *= np.float32(grow)
    return g


def _camera(W, H):
    return lonlat.Camera.from_view(scenes.make_view(W, H, (0.0, 0.0, 0.0), scenes.rotation_yaw_pitch(0.2, 0.1)))


@pytest.mark.parametrize("P,W,H,spread,grow", [
    # one pair per Gaussian and 4096 bins: lists of 128 n and 1024 n pairs and one to either side
    *[(P, 8192, 4096, 1e-4, 0.02) for P in (257, 383, 384, 385, 1023, 1024, 1025, 1152, 2049)],
    (40000, 8192, 4096, 0.001, 0.1),
    (60000, 2048, 1024, 0.02, 1.0), (200000, 2048, 1024, 0.2, 1.0), (200000, 2048, 1024, 0.002, 0.2),
    (13000, 2048, 1024, 0.0, 20.0),  # far more pairs than expected
    (5000, 2048, 1024, 0.0, 1.0), (5000, 2048, 1024, 0.05, 1.0), (3000, 2048, 1024, 0.0, 1.0), (9000, 2132, 1093, 0.0, 1.0),
    (300000, 64, 64, 0.0, 0.2), (100000, 200, 130, 0.1, 1.0)])
def test_lists_of_clustered_scenes(cuda, P, W, H, spread, grow):
    cu = helpers.run_cuda(lonlat.GaussianTensors.from_numpy(_clustered(P, spread, grow)), _camera(W, H))
    n = helpers.to_np
    b = oracle.binning(W, H, n(cu["radii"]), n(cu["means2D"]), n(cu["depths"]), None, f32=True)
    assert b["num_rendered"] == cu["num_rendered"] > 0
    np.testing.assert_array_equal(n(cu["tile_ids"]).view(np.uint32), (b["keys"] >> np.uint64(32)).astype(np.uint32))
    np.testing.assert_array_equal(n(cu["point_list"]).view(np.uint32), b["point_list"])
    np.testing.assert_array_equal(n(cu["ranges"]).view(np.uint32), b["ranges"])


@pytest.mark.parametrize("P,seam", [(30000, False), (30000, True), (7000, False)])
def test_lists_of_clustered_batches(cuda, P, seam):
    views = scenes.random_views(6, [(1024, 512), (500, 250), (2132, 1093), (64, 32)], seed=P)
    cams = batch.BatchCameras.from_views(views)
    gt = lonlat.GaussianTensors.from_numpy(_clustered(P, 0.05))
    _, per, state = batch.render_batch(gt, cams, seam_wrap=seam)
    helpers.check_batch_lists(state, cams, per, P, seam)


@pytest.mark.parametrize("P,W,H", [(3000, 2048, 1024), (5000, 2048, 1024), (1500, 512, 256), (13000, 8192, 4096)])
def test_captured_forward(cuda, P, W, H):
    gt, cam = lonlat.GaussianTensors.from_numpy(_clustered(P, 0.0)), _camera(W, H)
    image, radii, n, _ = lonlat.rasterize(gt, cam)
    state = lonlat.LonlatState(P, W, H, n)  # no instance to spare
    out, r = torch.empty_like(image), torch.empty_like(radii)
    state.forward(gt, cam, out, r)
    torch.cuda.synchronize()
    points = state.binning_view(n)["point_list"].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        state.forward(gt, cam, out, r)
    for _ in range(2):
        out.zero_()
        state.binning.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert state.status() == (n, 0)
        assert torch.equal(out, image) and torch.equal(r, radii)
        assert torch.equal(state.binning_view(n)["point_list"], points)


def _ranges_us(g, W, H):
    gt, cam = lonlat.GaussianTensors.from_numpy(g), _camera(W, H)
    image, radii, n, _ = lonlat.rasterize(gt, cam)
    state = lonlat.LonlatState(gt.P, W, H, n + n // 8)
    best = float("inf")
    for _ in range(8):
        torch.cuda.synchronize()
        capi.timing_enable(True)
        state.forward(gt, cam, image, radii)
        best = min(best, 1000 * capi.timing_read()["ranges"][0])
        capi.timing_enable(False)
    return best


@pytest.mark.parametrize("P,W,H,spread", [(1000000, 2048, 1024, 0.1), (1000000, 2048, 1024, 0.02)])
def test_cost_does_not_follow_the_spread(cuda, P, W, H, spread):
    # (a few warps with all of the pairs took 9 and 14 times as long as an even spread)
    assert _ranges_us(_clustered(P, spread), W, H) < 4.0 * _ranges_us(_clustered(P, 0.0), W, H)

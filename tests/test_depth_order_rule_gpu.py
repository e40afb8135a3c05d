"""The counted depth order of a batch on either side of its rule (at most 2^28 comparisons over the views, at most
12,288 Gaussians): lists bit-exact against the oracle, and ordering that many views costs no more than a depth sort
of as many Gaussians does."""
import pytest
import torch

import helpers
from omnigs_b200 import batch, capi, lonlat, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,V", [(5792, 8), (5793, 8), (2896, 32), (2897, 32), (12288, 3)])
def test_lists_on_either_side_of_the_rule(cuda, P, V):
    g = scenes.make_gaussians(P, seed=P)
    g.means3D[P // 2:] = g.means3D[:P - P // 2]  # equal depths: the index decides
    cams = batch.BatchCameras.from_views(scenes.random_views(V, [(128, 64), (65, 33)], seed=V))
    _, per, state = batch.render_batch(lonlat.GaussianTensors.from_numpy(g), cams)
    helpers.check_batch_lists(state, cams, per, P)


def _sort_us(P, V):
    """Best of several times of the sort stage of a batch (one launch when the order is counted)."""
    gt = lonlat.GaussianTensors.from_numpy(scenes.make_gaussians(P, seed=1))
    cams = batch.BatchCameras.from_views(scenes.random_views(V, [(64, 32)], seed=2))
    images, per, _ = batch.render_batch(gt, cams)
    state = batch.BatchState(P, cams.sizes, sum(per) + 1024)
    best = float("inf")
    for _ in range(8):
        torch.cuda.synchronize()
        capi.timing_enable(True)
        state.forward(gt, cams, images)
        best = min(best, 1000 * capi.timing_read()["sort"][0])
        capi.timing_enable(False)
    return best


def test_many_views_do_not_cost_more_than_the_sort(cuda):
    # 12,289 Gaussians are always sorted; counting 32 x 12,288 takes five times as long as sorting them
    assert _sort_us(12288, 32) < 2.0 * _sort_us(12289, 32)

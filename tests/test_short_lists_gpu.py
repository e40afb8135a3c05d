"""GPU tests of the forward blend's two kernels: the one for short lists is taken where the list's capacity bounds them,
so the same view with a tight and with a loose capacity runs both.  Images, transmittance and last contributors are
identical, also with some lists of many staging batches, splats on either side of the clamp, and non-finite ones."""
import numpy as np
import pytest
import torch

from omnigs_b200 import batch, capi, lonlat, scenes

pytestmark = pytest.mark.gpu


def _scene(P, clustered=False):
    g = scenes.make_gaussians(P, seed=P, seam_fraction=0.1)
    rng = np.random.default_rng(P)
    special = rng.random((P, 1)) < 0.3
    g.opacities[special] = rng.choice(np.float32([0.0, 0.003, 0.98, 0.98999, 0.99, 1.0]), int(special.sum()))
    if clustered:  # a third of them in a few tiles
        k = P // 3
        d = np.array([0.2, 0.1, 1.0]) + 0.01 * rng.standard_normal((k, 3))
        g.means3D[:k] = (3.0 * d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
        g.scales[:k] *= np.float32(0.1)
        g.opacities[:k] *= np.float32(0.05)
    return g


def _forward(gt, cam, capacity, recompute=False):
    P, W, H = gt.P, cam.width, cam.height
    state = lonlat.LonlatState(P, W, H, capacity, recompute_T=recompute)
    out, radii = torch.empty(3, H, W, device="cuda"), torch.empty(P, dtype=torch.int32, device="cuda")
    state.forward(gt, cam, out, radii)
    assert state.status()[1] == 0
    return out, state


def _loose(W, H):
    """A capacity above the short lists' rule."""
    return 50 * ((W + 15) // 16) * ((H + 15) // 16)


@pytest.mark.parametrize("P,W,H,clustered", [(1, 16, 16, False), (50, 100, 70, False), (3000, 1024, 512, False),
                                             (20000, 1520, 712, False), (20000, 2048, 1024, True)])
def test_both_kernels_agree(cuda, P, W, H, clustered):
    gt = lonlat.GaussianTensors.from_numpy(_scene(P, clustered))
    cam = lonlat.Camera.from_view(scenes.make_view(W, H, (0.0, 0.0, 0.0), scenes.rotation_yaw_pitch(0.1, 0.0)),
                                  background=(0.3, 0.2, 0.1))
    n = lonlat.rasterize(gt, cam)[2]
    loose = max(_loose(W, H), n)
    assert n < 40 * ((W + 15) // 16) * ((H + 15) // 16)
    a, sa = _forward(gt, cam, n)
    b, sb = _forward(gt, cam, loose)
    assert torch.equal(a, b)
    va, vb = sa.image_view(), sb.image_view()
    assert torch.equal(va["final_T"], vb["final_T"]) and torch.equal(va["n_contrib"], vb["n_contrib"])
    if clustered:
        ranges = va["ranges"].view(-1, 2)
        assert (ranges[:, 1] - ranges[:, 0]).max() > 3 * 128
    assert torch.equal(_forward(gt, cam, n, recompute=True)[0], a)


@pytest.mark.parametrize("seam", [False, True])
def test_both_kernels_agree_on_batches(cuda, seam):
    gt = lonlat.GaussianTensors.from_numpy(_scene(6000))
    cams = batch.BatchCameras.from_views(scenes.random_views(9, [(500, 250), (1024, 512), (33, 17), (256, 128)], seed=3))
    images, per, _ = batch.render_batch(gt, cams, seam_wrap=seam)
    outs = []
    for capacity in (sum(per), sum(_loose(w, h) for w, h in cams.sizes) + sum(per)):
        state = batch.BatchState(gt.P, cams.sizes, capacity)
        out = [torch.empty_like(i) for i in images]
        state.forward(gt, cams, out, seam_wrap=seam)
        outs.append(out)
    assert sum(per) < 40 * sum(((w + 15) // 16) * ((h + 15) // 16) for w, h in cams.sizes)
    assert all(torch.equal(a, b) for a, b in zip(*outs))


def test_non_finite_splats(cuda):
    """Indefinite and non-finite covariances, colours and opacities, at both kernels and both depth orders."""
    for P in (3000, 15000):
        g = _scene(P)
        gt = lonlat.GaussianTensors.from_numpy(g)
        rng = np.random.default_rng(7)
        cov = np.zeros((P, 6), np.float32)
        cov[:, [0, 3, 5]] = (g.scales.astype(np.float64) ** 2).astype(np.float32)
        odd = rng.permutation(P)[:200]
        cov[odd[:50], 1] = 10.0           # indefinite
        cov[odd[50:60], 3] = 1e12         # as wide as the image
        colors = rng.random((P, 3), np.float32)
        colors[odd[70:80], 0] = np.nan
        colors[odd[80:90], 1] = np.inf
        opacities = g.opacities.copy()
        opacities[odd[90:100]] = np.nan
        opacities[odd[100:110]] = np.inf
        opacities[odd[110:120]] = -np.inf
        means = g.means3D.copy()
        means[odd[120:130], 0] = np.nan
        means[odd[130:140], 1] = np.inf
        cov[odd[140:143], 0] = np.inf
        opacities[odd[50:60]] = opacities[odd[140:143]] = 0.02  # (they must not hide the others)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        gt = lonlat.GaussianTensors(t(means), t(opacities), colors_precomp=t(colors), cov3D_precomp=t(cov))
        W, H = 1024, 512
        cam = lonlat.Camera.from_view(scenes.make_view(W, H, (0.0, 0.0, 0.0), scenes.rotation_yaw_pitch(0.1, 0.0)))
        image, radii, n, state = lonlat.rasterize(gt, cam)
        a, _ = _forward(gt, cam, n)
        b, sb = _forward(gt, cam, n + _loose(W, H))
        eq = lambda x, y: torch.equal(x.view(torch.int32), y.view(torch.int32))  # noqa: E731
        nan_eq = lambda x, y: torch.equal(torch.nan_to_num(x, 7.0), torch.nan_to_num(y, 7.0))  # noqa: E731
        assert nan_eq(a, b)
        assert bool(torch.isnan(a).any()) and not bool(torch.isnan(a).all())
        assert eq(sb.image_view()["final_T"], state.image_view()["final_T"])


def test_short_lists_cost_less_with_their_kernel(cuda):
    P, W, H = 20000, 2048, 1024  # 2.4 Gaussians and 21 instances a tile
    gt = lonlat.GaussianTensors.from_numpy(scenes.make_gaussians(P, seed=1))
    cam = lonlat.Camera.from_view(scenes.make_view(W, H, (0.2, 0.1, 0.0), scenes.rotation_yaw_pitch(0.1, 0.0)))
    n = lonlat.rasterize(gt, cam)[2]
    out, radii = torch.empty(3, H, W, device=cuda), torch.empty(P, dtype=torch.int32, device=cuda)

    def best(capacity):
        state, t = lonlat.LonlatState(P, W, H, capacity), float("inf")
        for _ in range(20):
            torch.cuda.synchronize()
            capi.timing_enable(True)
            state.forward(gt, cam, out, radii)
            t = min(t, capi.timing_read()["render_forward"][0])
            capi.timing_enable(False)
        return t

    assert best(n) < 0.99 * best(_loose(W, H))

"""Performance cases of the equirectangular rasterizer and of the training step around it.

``listed()`` names the cases that are timed, ``draw()`` gives more of the same ranges, ``prepare()``
makes what a program holds before the call (scene, camera, state buffers, all on the GPU, from a
seed alone), ``run()`` is one pass through the public entry points, ``work()`` the bytes and
operations that a pass cannot do without and ``exact()`` its outputs in 64 bits, from plain torch.

Kinds of cases:

* ``train_view``: forward + backward of one view through ``GaussianRasterizer`` (LibTorch autograd),
  what a drop-in trainer does for every keyframe;
* ``render_view``: the forward of one view through ``LonlatState``, what a viewer or an evaluation
  over held-out views does;
* ``batch``: forward + backward of several views of uneven size in one call (``BatchState``), with
  BF16 SH, FP64 poles or seam wrapping where a program asks for them;
* ``loss``: L1 + D-SSIM and its image gradient (``train.l1_dssim``), once per view and iteration;
* ``adam``: the fused parameter update (``GaussianModelState.adam_step``), once per iteration;
* ``train_step``: a whole iteration over a batch (``BatchTrainStep``), captured once and replayed.

Scenes have the distributions of ``omnigs_b200.scenes`` (a shell of radius 1 to 5 around the cameras),
made on the GPU so that large ones are quick.
"""
from __future__ import annotations

import math

import torch

SHELL = (1.0, 5.0)


# ------------------------------------------------------------------------------------- cases ---
def listed() -> list:
    return [
        # the smallest training views: the finite-difference subset of the differentiation workload
        # and the CPU-runnable workload; launches and latency count
        dict(name="train_view_1k", kind="train_view", P=1000, W=256, H=128, degree=3),
        dict(name="train_view_10k", kind="train_view", P=10000, W=512, H=256, degree=3),
        # a panorama of the size published for the 360Roam captures: neither side a multiple of the
        # tile, SH degree 2 (a trainer raises the degree from 0 to 3 while it runs)
        dict(name="train_view_300k", kind="train_view", P=300000, W=1520, H=712, degree=2),
        # the headline view
        dict(name="train_view_1m", kind="train_view", P=1000000, W=2048, H=1024, degree=3),
        # the largest view: the peak-memory workload
        dict(name="train_view_3m", kind="train_view", P=3000000, W=4096, H=2048, degree=3),
        # rendering only: a small preview and the headline view
        dict(name="render_view_10k", kind="render_view", P=10000, W=512, H=256, degree=3),
        dict(name="render_view_1m", kind="render_view", P=1000000, W=2048, H=1024, degree=3),
        # the batched workload: 16 views of four resolutions over one scene, SH stored as BF16
        dict(name="batch_16_views", kind="batch", P=1000000, V=16, sizes="mixed", W=2048, H=1024, degree=3,
             bf16=True, poles=False, seam=False, pole_fraction=0.0),
        # the precision mode on a pole-heavy scene
        dict(name="batch_poles", kind="batch", P=300000, V=1, sizes="same", W=2048, H=1024, degree=3,
             bf16=True, poles=True, seam=False, pole_fraction=0.3),
        # the photometric loss of one headline image
        dict(name="loss_2048x1024", kind="loss", W=2048, H=1024, rows=1024),
        # the parameter update of the headline scene
        dict(name="adam_1m", kind="adam", P=1000000, M=16, bf16=False),
        # a whole training iteration over a few views, captured in a CUDA graph
        dict(name="train_step_4_views", kind="train_step", P=200000, V=4, sizes="mixed", W=1024, H=512, degree=3,
             bf16=True),
    ]


def _log_int(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["train_view"] * 5 + ["render_view"] * 2 + ["batch"] * 2 + ["loss", "adam", "train_step"])
    if kind == "adam":
        return dict(kind=kind, P=_log_int(rng, 1000, 2000000), M=rng.choice([1, 4, 9, 16, 16, 16]),
                    bf16=rng.random() < 0.5)
    # about twice as wide as high, any parity
    H = _log_int(rng, 128, 2048 if kind in ("train_view", "render_view") else 1024)
    W = 2 * H if rng.random() < 0.4 else int(round(H * rng.uniform(1.8, 2.2)))
    if W > 4096:
        W = 4096
    if kind == "loss":
        H, W = 2 * H, min(2 * W, 4096)
        return dict(kind=kind, W=W, H=H, rows=H if rng.random() < 0.6 else max(1, int(H * rng.uniform(0.7, 1.0))))
    density = math.exp(rng.uniform(math.log(0.03), math.log(0.7)))  # Gaussians per pixel
    P = max(500, min(3000000, int(W * H * density)))
    degree = rng.choice([0, 1, 2, 3, 3, 3])
    if kind in ("train_view", "render_view"):
        return dict(kind=kind, P=P, W=W, H=H, degree=degree)
    P = min(P, 400000)
    V = rng.randint(1, 6) if kind == "batch" else rng.randint(1, 4)
    sizes = rng.choice(["mixed", "same"])
    if kind == "train_step":
        return dict(kind=kind, P=P, V=V, sizes=sizes, W=W, H=H, degree=3, bf16=rng.random() < 0.5)
    option = rng.choice(["none", "none", "poles", "seam"])
    return dict(kind=kind, P=P if option != "poles" else min(P, 100000), V=V if option != "poles" else min(V, 2),
                sizes=sizes, W=W, H=H, degree=degree, bf16=rng.random() < 0.5, poles=option == "poles",
                seam=option == "seam", pole_fraction=0.3 if option == "poles" else 0.0)


def view_sizes(case) -> list:
    """(W, H) of the case's views; "mixed" cycles through 1/4, 1/2, 1 and 3/2 of the given size, as
    the batched workload's {512x256, 1024x512, 2048x1024, 3072x1536} for 2048x1024."""
    V = case.get("V", 1)
    if case.get("sizes", "same") == "same":
        return [(case["W"], case["H"])] * V
    num, den = (1, 1, 1, 3), (4, 2, 1, 2)
    order = (1, 2, 3, 2, 1, 1, 1, 3, 1, 3, 1, 0, 1, 0, 1, 3)  # the mix of the batched workload
    return [(max(16, case["W"] * num[k] // den[k]), max(16, case["H"] * num[k] // den[k]))
            for k in (order[v % 16] for v in range(V))]


# ------------------------------------------------------------------------------------ inputs ---
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _scene(case, gen) -> dict:
    """Activated parameters of the scene, float32 on the GPU."""
    P = case["P"]
    n = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    u = lambda *s: torch.rand(*s, generator=gen, device="cuda")  # noqa: E731
    lo, hi = SHELL
    r = (u(P, 1) * (hi ** 3 - lo ** 3) + lo ** 3) ** (1.0 / 3.0)
    d = torch.nn.functional.normalize(n(P, 3), dim=1)
    frac = case.get("pole_fraction", 0.0)
    if frac > 0:  # that share of the means beyond 80 degrees of latitude
        s0 = math.sin(math.radians(80.0))
        sin_lat = (s0 + (1.0 - s0) * u(P)) * torch.where(u(P) < 0.5, -1.0, 1.0)
        lon = (2.0 * u(P) - 1.0) * math.pi
        cos_lat = torch.sqrt(1.0 - sin_lat * sin_lat)
        polar = torch.stack([cos_lat * torch.sin(lon), sin_lat, cos_lat * torch.cos(lon)], 1)
        d = torch.where((u(P) < frac)[:, None], polar, d)
    shs = 0.05 * n(P, 16, 3)
    shs[:, 0] *= 10.0
    return dict(means=(d * r).contiguous(), scales=torch.exp(math.log(0.02) + 0.5 * n(P, 3)),
                rotations=torch.nn.functional.normalize(n(P, 4), dim=1), opacities=torch.sigmoid(n(P, 1)), shs=shs)


def _cameras(case, gen) -> tuple:
    """viewmatrices [V,4,4] (row-major Tcw^T), camera centres [V,3] and backgrounds [V,3]: positions in a
    2 m cube, any yaw, pitch within 30 degrees; pole-heavy scenes are seen from the origin, upright, so
    that their poles are the image's."""
    V = case.get("V", 1)
    u = torch.rand(V, 8, generator=gen, device="cuda").cpu().double()
    vms, centres = [], []
    for v in range(V):
        if case.get("pole_fraction", 0.0) > 0:
            c, yaw, pitch = 0.02 * (u[v, :3] - 0.5), 0.0, 0.0
        else:
            c = 2.0 * (u[v, :3] - 0.5)
            yaw, pitch = float(2 * u[v, 3] - 1) * math.pi, math.radians(30.0) * float(2 * u[v, 4] - 1)
        cy, sy, cp, sp = math.cos(yaw), math.sin(yaw), math.cos(pitch), math.sin(pitch)
        Ry = torch.tensor([[cy, 0, sy], [0, 1, 0], [-sy, 0, cy]], dtype=torch.float64)
        Rx = torch.tensor([[1, 0, 0], [0, cp, -sp], [0, sp, cp]], dtype=torch.float64)
        R = (Ry @ Rx).T
        T = torch.eye(4, dtype=torch.float64)
        T[:3, :3] = R
        T[:3, 3] = -R @ c
        vms.append(T.T)
        centres.append(c)
    f = lambda t: t.float().cuda().contiguous()  # noqa: E731
    return f(torch.stack(vms)), f(torch.stack(centres)), f(0.3 * u[:, 5:8])


def _upstream(case, gen) -> list:
    return [torch.randn(3, h, w, generator=gen, device="cuda") for w, h in view_sizes(case)]


def _view_inputs(case, seed) -> tuple:
    gen = _generator(seed)
    scene = _scene(case, gen)
    if case.get("bf16"):
        scene["shs"] = scene["shs"].bfloat16()
    cams = _cameras(case, gen)
    return scene, cams, _upstream(case, gen)


def _images(case, seed) -> tuple:
    """A rendered-looking image and its target: smooth colour fields, the first with more noise."""
    gen = _generator(seed)
    H, W = case["H"], case["W"]
    low = torch.rand(1, 3, max(2, H // 24), max(2, W // 24), generator=gen, device="cuda")
    gt = torch.nn.functional.interpolate(low, size=(H, W), mode="bilinear", align_corners=False)[0]
    gt = (gt + 0.02 * torch.randn(3, H, W, generator=gen, device="cuda")).clamp(0, 1).contiguous()
    img = (gt + 0.05 * torch.randn(3, H, W, generator=gen, device="cuda")).clamp_min(0).contiguous()
    return img, gt


def _adam_inputs(case, seed) -> tuple:
    """Raw parameters, in the order of the optimizer's groups, and gradients of a few 1e-4."""
    gen = _generator(seed)
    P, M = case["P"], case["M"]
    n = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    raw = [2.0 * n(P, 3), 0.5 * n(P, 1, 3), 0.05 * n(P, M - 1, 3), n(P, 1), math.log(0.02) + 0.5 * n(P, 3), n(P, 4)]
    grads = [1e-4 * n(P, 3), 1e-4 * n(P, M, 3), 1e-4 * n(P, 1), 1e-3 * n(P, 3), 1e-4 * n(P, 4)]
    return raw, grads


# late-training learning rates: a step changes the scene, and with it the next pass's work, little
STEP_LR = dict(xyz=1.6e-6, f_dc=2.5e-4, f_rest=1.25e-5, opacity=5e-3, scaling=5e-4, rotation=1e-4)


# --------------------------------------------------------------------------- prepare and run ---
def prepare(case, seed) -> dict:
    import omnigs_b200
    from omnigs_b200 import batch, lonlat, train

    kind = case["kind"]
    s = dict(kind=kind)
    if kind == "loss":
        img, gt = _images(case, seed)
        return dict(s, img=img, gt=gt, rows=case["rows"], dimg=torch.empty_like(img),
                    loss=torch.empty(3, device="cuda"), ws=train.l1_dssim_workspace(3, case["H"], case["W"]))
    if kind == "adam":
        raw, grads = _adam_inputs(case, seed)
        return dict(s, model=train.GaussianModelState(*raw, sh_bf16=case["bf16"]), grads=grads)
    scene, (vms, centres, bgs), dimages = _view_inputs(case, seed)
    sizes = view_sizes(case)
    if kind == "train_view":
        leaf = {k: t.requires_grad_(True) for k, t in scene.items()}
        leaf["means2D"] = torch.zeros_like(scene["means"]).requires_grad_(True)
        (w, h), = sizes
        settings = omnigs_b200.GaussianRasterizationSettings(h, w, 0.0, 0.0, bgs[0], 1.0, vms[0], vms[0],
                                                             case["degree"], centres[0])
        return dict(s, rasterizer=omnigs_b200.GaussianRasterizer(settings), leaf=leaf, dimage=dimages[0])
    gt = lonlat.GaussianTensors(scene["means"], scene["opacities"], scene["shs"], scene["scales"], scene["rotations"])
    if kind == "render_view":
        (w, h), = sizes
        cam = lonlat.Camera(w, h, vms[0], centres[0], bgs[0])
        n = lonlat.rasterize(gt, cam, D=case["degree"])[2]
        return dict(s, g=gt, cam=cam, D=case["degree"], state=lonlat.LonlatState(gt.P, w, h, n + n // 8 + 1024),
                    out=torch.empty(3, h, w, device="cuda"),
                    radii=torch.empty(gt.P, dtype=torch.int32, device="cuda"))
    cams = batch.BatchCameras(sizes, vms, centres, bgs)
    options = dict(fp64_poles=case.get("poles", False), seam_wrap=case.get("seam", False))
    images, per, st = batch.render_batch(gt, cams, D=case["degree"], **options)
    n = sum(per)
    if kind == "batch":
        return dict(s, g=gt, cams=cams, D=case["degree"], options=options, images=images, dimages=dimages,
                    state=batch.BatchState(gt.P, sizes, n + n // 8 + 1024),
                    grads=batch.BatchGradients.empty(gt.P, gt.M, "cuda"))
    del st
    # targets: the scene's own views; the model starts a little off them
    gen = _generator(int(seed) + 1)
    logit = lambda o: torch.log(o / (1 - o))  # noqa: E731
    sh = scene["shs"].float()
    sh = sh + 0.02 * torch.randn(sh.shape, generator=gen, device="cuda")
    means = scene["means"] + 0.003 * torch.randn(scene["means"].shape, generator=gen, device="cuda")
    model = train.GaussianModelState(means, sh[:, :1], sh[:, 1:], logit(scene["opacities"].clamp(1e-6, 1 - 1e-6)),
                                     torch.log(scene["scales"]), scene["rotations"], sh_bf16=case["bf16"], lr=STEP_LR)
    step = train.BatchTrainStep(model, cams, images, n + n // 4 + 1024, D=case["degree"])
    step.run()
    step.capture()
    return dict(s, step=step)


def run(state):
    kind = state["kind"]
    if kind == "train_view":
        t = state["leaf"]
        color, radii = state["rasterizer"](t["means"], t["means2D"], t["opacities"], shs=t["shs"], scales=t["scales"],
                                           rotations=t["rotations"])
        names = ("means", "means2D", "opacities", "shs", "scales", "rotations")
        grads = torch.autograd.grad([color], [t[k] for k in names], [state["dimage"]])
        return dict(color=color.detach(), radii=radii, **{"d_" + k: g for k, g in zip(names, grads)})
    if kind == "render_view":
        state["state"].forward(state["g"], state["cam"], state["out"], state["radii"], D=state["D"])
        return dict(color=state["out"], radii=state["radii"])
    if kind == "batch":
        st, g, cams, D, opt = (state[k] for k in ("state", "g", "cams", "D", "options"))
        st.forward(g, cams, state["images"], D=D, **opt)
        st.backward(g, cams, state["dimages"], state["grads"], D=D, **opt)
        return dict(images=list(state["images"]), **_grads(state["grads"]))
    if kind == "loss":
        from omnigs_b200 import train
        loss, d = train.l1_dssim(state["img"], state["gt"], 0.2, rows=state["rows"], dL_dimage=state["dimg"],
                                 loss=state["loss"], workspace=state["ws"])
        return dict(loss=loss, d_image=d)
    if kind == "adam":
        m = state["model"]
        m.adam_step(*state["grads"])
        return dict(params=list(m.params), m=list(m.m), v=list(m.v), shs=m.shs, opacities=m.opacities,
                    scales=m.scales, rotations=m.rotations)
    step = state["step"]
    step.replay()
    return dict(losses=step.losses, images=list(step.images), m=list(step.model.m), **_grads(step.grads))


def _grads(g) -> dict:
    return dict(d_means=g.dL_dmeans3D, d_shs=g.dL_dsh, d_opacities=g.dL_dopacity, d_scales=g.dL_dscales,
                d_rotations=g.dL_drotations)


# -------------------------------------------------------------------------------------- work ---
def work(case) -> dict:
    """Inputs read once and outputs written once; operations of the blends from the area of a splat.

    Mean area of a splat's support (alpha >= 1/255) in pixels: 2 pi E[ln(255 o)] times E[sx sy], with
    E[s s'] = 0.02^2 e^0.25, E[1 / r^2] over the shell, W / (2 pi) by H / pi pixels a radian and E[1 / cos(latitude)]
    = pi / 2 across.  About 25 operations a (pixel, splat) pair forward and 45 backward; a pixel is done
    after some 400 of them at most."""
    kind = case["kind"]
    if kind == "loss":
        n = 3 * case["W"] * case["rows"]
        return dict(bytes=4 * (2 * n + 3 * case["W"] * case["H"]), flops=(5 + 3) * 2 * 2 * 11 * n)
    if kind == "adam":
        per = 3 * case["M"] + 11
        return dict(bytes=case["P"] * (28 * per + (2 if case["bf16"] else 4) * (per - 3)), flops=16 * per * case["P"])
    lo, hi = SHELL
    inv_r2 = 3.0 * (hi - lo) / (hi ** 3 - lo ** 3)
    backward = kind != "render_view"
    sh = 96 if case.get("bf16") else 192
    P = case["P"]
    nbytes, flops = P * (44 + sh) + (P * (44 + 192) if backward else 0), 0.0
    for w, h in view_sizes(case):
        area = 2 * math.pi * 4.7 * (0.0004 * math.exp(0.25) * inv_r2 * w * h * math.pi / 2 / (2 * math.pi ** 2) + 0.3)
        pairs = min(P * area, 400.0 * w * h)
        nbytes += 12 * w * h * (2 if backward else 1) + 4 * P
        flops += pairs * (70 if backward else 25)
    if kind == "train_step":
        params = 59 * P
        nbytes += 28 * params + sum(12 * w * h for w, h in view_sizes(case))
        flops += 16 * params + sum((5 + 3) * 2 * 2 * 11 * 3 * w * h for w, h in view_sizes(case))
    return dict(bytes=int(nbytes), flops=int(flops))


# ------------------------------------------------------------------------------------- exact ---
def _sh_color(degree, dirs, sh):
    x, y, z = dirs.unbind(1)
    xx, yy, zz, xy, yz, xz = x * x, y * y, z * z, x * y, y * z, x * z
    b = [torch.full_like(x, 0.28209479177387814)]
    if degree > 0:
        b += [-0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x]
    if degree > 1:
        b += [1.0925484305920792 * xy, -1.0925484305920792 * yz, 0.31539156525252005 * (2 * zz - xx - yy),
              -1.0925484305920792 * xz, 0.5462742152960396 * (xx - yy)]
    if degree > 2:
        b += [-0.5900435899266435 * y * (3 * xx - yy), 2.890611442640554 * xy * z,
              -0.4570457994644658 * y * (4 * zz - xx - yy), 0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy),
              -0.4570457994644658 * x * (4 * zz - xx - yy), 1.445305721320277 * z * (xx - yy),
              -0.5900435899266435 * x * (xx - 3 * yy)]
    basis = torch.stack(b, 1)
    return (torch.einsum("pk,pkc->pc", basis, sh[:, :basis.shape[1]]) + 0.5).clamp_min(0.0)


def _project(t, vm, centre, W, H, degree):
    """Pixel centre, conic (a, b, c), colour, distance and radius of every Gaussian, in 64 bits."""
    p = t["means"] @ vm[:3, :3] + vm[3, :3]
    x, y, z = p.unbind(1)
    r = p.norm(dim=1)
    pix = torch.stack([((torch.atan2(x, z) / math.pi + 1) * W - 1) * 0.5,
                       ((torch.asin(y / (r + 1e-7)) * 2 / math.pi + 1) * H - 1) * 0.5], 1)
    q0, q1, q2, q3 = t["rotations"].unbind(1)
    R = torch.stack([1 - 2 * (q2 * q2 + q3 * q3), 2 * (q1 * q2 - q0 * q3), 2 * (q1 * q3 + q0 * q2),
                     2 * (q1 * q2 + q0 * q3), 1 - 2 * (q1 * q1 + q3 * q3), 2 * (q2 * q3 - q0 * q1),
                     2 * (q1 * q3 - q0 * q2), 2 * (q2 * q3 + q0 * q1), 1 - 2 * (q1 * q1 + q2 * q2)], 1).view(-1, 3, 3)
    L = R * t["scales"][:, None, :]
    rho2 = x * x + z * z
    rho = rho2.sqrt()
    i2, i1, ir = 1 / (rho2 + 1e-7), 1 / (rho + 1e-7), 1 / (rho2 + y * y + 1e-7)
    kw, kh = W * 0.5 / math.pi, H / math.pi
    zero = torch.zeros_like(x)
    J = torch.stack([kw * z * i2, zero, -kw * x * i2,
                     -kh * x * y * i1 * ir, kh * rho * ir, -kh * z * y * i1 * ir], 1).view(-1, 2, 3)
    A = J @ (vm[:3, :3].T @ L)
    cov = A @ A.transpose(1, 2)
    a, b, c = cov[:, 0, 0] + 0.3, cov[:, 0, 1], cov[:, 1, 1] + 0.3
    det = a * c - b * b
    conic = torch.stack([c / det, -b / det, a / det], 1)
    mid = 0.5 * (a + c)
    radius = torch.ceil(3 * torch.sqrt(mid + torch.sqrt((mid * mid - det).clamp_min(0.1)))).detach()
    d = t["means"] - centre
    color = _sh_color(degree, d / d.norm(dim=1, keepdim=True), t["shs"])
    return pix, conic, color, r.detach(), radius


def _exact_view(t, vm, centre, bg, dimage, W, H, degree, seam):
    """Image, and the gradients of (image . dimage) by the scene's tensors and the pixel centres, of one view."""
    pix, conic, color, dist, radius = _project(t, vm, centre, W, H, degree)
    gx, gy = (W + 15) // 16, (H + 15) // 16
    xy = pix.detach()
    # tile rects as the rasterizer clamps them (truncated towards zero)
    x0 = ((xy[:, 0] - radius) / 16).trunc().clamp(0, gx)
    x1 = ((xy[:, 0] + radius + 15) / 16).trunc().clamp(0, gx)
    y0 = ((xy[:, 1] - radius) / 16).trunc().clamp(0, gy)
    y1 = ((xy[:, 1] + radius + 15) / 16).trunc().clamp(0, gy)
    seen = (dist * dist > 0.04) & (x1 > x0) & (y1 > y0)
    order = torch.argsort(dist)
    order = order[seen[order]]
    x0, x1, y0, y1 = x0[order], x1[order], y0[order], y1[order]
    leaf = [v.detach() for v in (pix, conic, color, t["opacities"])]
    acc = [torch.zeros_like(v) for v in leaf]
    image = torch.empty(3, H, W, dtype=torch.float64, device="cuda")
    for ty in range(gy):
        in_row = ((y0 <= ty) & (y1 > ty)).nonzero()[:, 0]
        rx0, rx1, rid = x0[in_row], x1[in_row], order[in_row]
        py = torch.arange(16 * ty, min(16 * ty + 16, H), device="cuda", dtype=torch.float64)
        for tx in range(gx):
            px = torch.arange(16 * tx, min(16 * tx + 16, W), device="cuda", dtype=torch.float64)
            idx = rid[(rx0 <= tx) & (rx1 > tx)]
            ys, xs = slice(16 * ty, 16 * ty + len(py)), slice(16 * tx, 16 * tx + len(px))
            if idx.numel() == 0:
                image[:, ys, xs] = bg[:, None, None]
                continue
            m, q, c, o = (v[idx].requires_grad_(True) for v in leaf)
            dx = m[:, :1] - px.repeat(len(py))[None]
            dy = m[:, 1:] - py.repeat_interleave(len(px))[None]
            power = -0.5 * (q[:, :1] * dx * dx + q[:, 2:] * dy * dy) - q[:, 1:2] * dx * dy
            full = o * torch.exp(power)
            alpha = full - (full - full.clamp_max(0.99)).detach()  # the gradient passes the clamp
            alpha = torch.where((power <= 0) & (alpha >= 1 / 255), alpha, torch.zeros_like(alpha))
            after = torch.cumprod(1 - alpha, 0)
            live = after >= 1e-4  # a pixel stops at the splat that would take it below
            alpha = alpha * live
            after = torch.cumprod(1 - alpha, 0)
            before = torch.cat([torch.ones_like(after[:1]), after[:-1]], 0)
            col = torch.einsum("np,nc->cp", alpha * before, c) + bg[:, None] * after[-1]
            image[:, ys, xs] = col.detach().view(3, len(py), len(px))
            if dimage is not None:
                g = torch.autograd.grad((col * dimage[:, ys, xs].reshape(3, -1)).sum(), (m, q, c, o))
                for a, v in zip(acc, g):
                    a.index_add_(0, idx, v)
    if dimage is None:
        return image, None, None
    names = ("means", "shs", "scales", "rotations")
    g = torch.autograd.grad([pix, conic, color], [t[k] for k in names], acc[:3])
    grads = dict(zip(names, g), opacities=acc[3])
    scale = torch.tensor([0.5 * W, 0.5 * H], dtype=torch.float64, device="cuda")
    return image, grads, torch.cat([acc[0] * scale, torch.zeros_like(acc[0][:, :1])], 1)


# tiles and (Gaussian, view) records up to which the 64-bit rendering stays within seconds
EXACT_TILES, EXACT_RECORDS = 4500, 400000


def _exact_views(case, seed):
    sizes = view_sizes(case)
    tiles = sum(((w + 15) // 16) * ((h + 15) // 16) for w, h in sizes)
    if tiles > EXACT_TILES or case["P"] * len(sizes) > EXACT_RECORDS or case.get("seam"):
        return None
    scene, (vms, centres, bgs), dimages = _view_inputs(case, seed)
    backward = case["kind"] != "render_view"
    t = {k: v.double().requires_grad_(True) for k, v in scene.items()}
    images, total, d2 = [], None, None
    for v, (w, h) in enumerate(sizes):
        im, g, d2 = _exact_view(t, vms[v].double(), centres[v].double(), bgs[v].double(),
                                dimages[v].double() if backward else None, w, h, case["degree"], False)
        images.append(im)
        total = g if total is None else {k: total[k] + g[k] for k in g}
    if case["kind"] == "render_view":
        return dict(color=images[0], radii=None)
    if case["kind"] == "train_view":
        return dict(color=images[0], radii=None, d_means2D=d2, **{"d_" + k: g for k, g in total.items()})
    return dict(images=images, **{"d_" + k: g for k, g in total.items()})


def _exact_loss(case, seed):
    img, gt = (t.double() for t in _images(case, seed))
    rows = case["rows"]
    w = torch.exp(-(torch.arange(11, dtype=torch.float64, device="cuda") - 5) ** 2 / (2 * 1.5 ** 2))
    w = w / w.sum()
    img = img.requires_grad_(True)
    a, b = img[None, :, :rows], gt[None, :, :rows]

    def blur(v):
        v = torch.nn.functional.conv2d(v, w.view(1, 1, 1, 11).expand(3, 1, 1, 11), padding=(0, 5), groups=3)
        return torch.nn.functional.conv2d(v, w.view(1, 1, 11, 1).expand(3, 1, 11, 1), padding=(5, 0), groups=3)

    m1, m2 = blur(a), blur(b)
    s1, s2, s12 = blur(a * a) - m1 * m1, blur(b * b) - m2 * m2, blur(a * b) - m1 * m2
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    ssim = (((2 * m1 * m2 + c1) * (2 * s12 + c2)) / ((m1 * m1 + m2 * m2 + c1) * (s1 + s2 + c2))).mean()
    l1 = (a - b).abs().mean()
    loss = 0.8 * l1 + 0.2 * (1 - ssim)
    d, = torch.autograd.grad(loss, img)
    return dict(loss=torch.stack([loss, l1, ssim]).detach(), d_image=d)


def _exact_adam(case, seed):
    raw, grads = _adam_inputs(case, seed)
    raw, grads = [t.double() for t in raw], [t.double() for t in grads]
    d_xyz, d_sh, d_op, d_sc, d_rot = grads
    o, e, q = torch.sigmoid(raw[3]), torch.exp(raw[4]), raw[5]
    n = q.norm(dim=1, keepdim=True)
    y = q / n
    g = [d_xyz, d_sh[:, :1], d_sh[:, 1:], d_op * o * (1 - o), d_sc * e, (d_rot - y * (y * d_rot).sum(1, keepdim=True)) / n]
    lr = (0.00016, 0.0025, 0.0025 / 20.0, 0.05, 0.005, 0.001)
    b1, b2, eps = 0.9, 0.999, 1e-15
    m, v = [(1 - b1) * t for t in g], [(1 - b2) * t * t for t in g]
    p = [t - k / (1 - b1) * mm / ((vv / (1 - b2)).sqrt() + eps) for t, k, mm, vv in zip(raw, lr, m, v)]
    return dict(params=p, m=m, v=v, shs=torch.cat([p[1], p[2]], 1), opacities=torch.sigmoid(p[3]),
                scales=torch.exp(p[4]), rotations=p[5] / p[5].norm(dim=1, keepdim=True))


def exact(case, seed):
    kind = case["kind"]
    if kind == "loss":
        return _exact_loss(case, seed)
    if kind == "adam":
        return _exact_adam(case, seed)
    if kind == "train_step":
        return None
    return _exact_views(case, seed)

"""The work that users of this library have it do, as timed cases.

Each case is one call (or one short call sequence) through the public Python
API on inputs of the shape, type and distribution that the call meets in use:

* ``pair``: a whole stereo pair, frame stacks in, organised cloud out;
* ``decode``: one camera's fringe stack to fringe orders and phase;
* ``rectify_match``: two decoded cameras to a disparity map (one call);
* ``reconstructor``: the reference-shaped class, setData + startCalculate with
  its default configuration (rectify, match, median, reprojection, pixel
  Gaussian, radius outlier filter);
* ``sor``, ``mls``, ``metric_gaussian``: one point-cloud filter each;
* ``diff_backward``: one step of calibration refinement (forward + adjoint).

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges.
``exact(case, seed)`` restates a case's outputs in 64 bits with plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from zim_gb300 import api, diff, synth

TWO_PI = 2.0 * math.pi
PLANE_Z = 900.0          # mm, the scenes' background plane


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------
def listed():
    return [
        # the smallest whole call: one VGA pair, Gray code, SOR; bound by launches and latency
        dict(name="pair_gray_u8_640x480", kind="pair", encoding="gray", width=640, height=480, mean_k=50,
             smooth=False),
        # the library's main workload: a 5 MP 12-bit pair through every stage and the smoothing filters
        dict(name="pair_hier_u16_2448x2048", kind="pair", encoding="hier", width=2448, height=2048, mean_k=30,
             smooth=True),
        # the reference's own default decoder: heterodyne 121/110/120, eight steps, 8-bit, 24 frames of a 5 MP camera
        dict(name="decode_heterodyne_u8_2448x2048", kind="decode", encoding="hetero", width=2448, height=2048,
             hdr=False),
        # a cropped sensor, whose rows are no multiple of 16 bytes; Gray code, ten frames
        dict(name="decode_gray_u8_1626x1236", kind="decode", encoding="gray", width=1626, height=1236, hdr=False),
        # shiny parts: the HDR least-squares decode of a 1.3 MP heterodyne stack with saturated pixels
        dict(name="decode_hdr_u8_1280x1024", kind="decode", encoding="hetero", width=1280, height=1024, hdr=True),
        # the step between two decoded 5 MP cameras and their disparity map
        dict(name="rectify_match_2448x2048", kind="rectify_match", width=2448, height=2048),
        # the drop-in class with its default configuration on the largest camera (12 MP)
        dict(name="reconstructor_4096x3000", kind="reconstructor", width=4096, height=3000, radius=0.7),
        # outlier removal on its own, with a k that is neither of the two workloads' values
        dict(name="sor_k20_1280x1024", kind="sor", width=1280, height=1024, mean_k=20),
        # the reference's default MLS parameters (order 1, 61 x 61 window, sigma 0.6 mm, three passes) on a 5 MP cloud
        dict(name="mls_default_2448x2048", kind="mls", width=2448, height=2048, order=1, window=30, sigma=0.6,
             radius=0.0, iterations=3),
        # second-order MLS within 2 mm on a 2 MP cloud
        dict(name="mls_order2_1626x1236", kind="mls", width=1626, height=1236, order=2, window=7,
             sigma=2.0 / math.sqrt(2.0), radius=2.0, iterations=1),
        # the last smoothing step of a 1.3 MP cloud
        dict(name="metric_gaussian_1280x1024", kind="metric_gaussian", width=1280, height=1024, sigma=0.5),
        # calibration refinement: one forward + adjoint over four poses of a planar target at 5 MP
        dict(name="diff_backward_4x2448x2048", kind="diff_backward", width=2448, height=2048, poses=4),
    ]


def _draw_size(rng, lo_w, hi_w):
    """A camera size: width log-uniform in [lo_w, hi_w], 4:3 to 5:4, odd ones among them."""
    w = int(round(math.exp(rng.uniform(math.log(lo_w), math.log(hi_w)))))
    if rng.random() < 0.5:
        w -= w % 16  # sensors mostly have round widths
    h = int(w * rng.uniform(0.73, 0.8))
    return w, h


def draw(rng):
    kind = rng.choice(["pair", "pair", "decode", "decode", "decode", "rectify_match", "reconstructor", "sor", "mls",
                       "mls", "metric_gaussian", "diff_backward"])
    if kind == "pair":
        w, h = _draw_size(rng, 640, 2448)
        return dict(kind=kind, encoding=rng.choice(["gray", "hier"]), width=w, height=h, mean_k=rng.choice([30, 50]),
                    smooth=rng.random() < 0.5)
    if kind == "decode":
        w, h = _draw_size(rng, 640, 2448)
        enc = rng.choice(["gray", "hier", "hetero"])
        return dict(kind=kind, encoding=enc, width=w, height=h, hdr=enc != "gray" and rng.random() < 0.3)
    if kind == "rectify_match":
        w, h = _draw_size(rng, 640, 2448)
    elif kind == "reconstructor":
        w, h = _draw_size(rng, 640, 4000)
        # the outlier radius goes with the camera's pixel spacing: the default 0.7 mm is three pixels of the 12 MP one
        return dict(kind=kind, width=w, height=h, radius=0.7 * 4096 / w)
    elif kind == "sor":
        w, h = _draw_size(rng, 640, 1280)
        return dict(kind=kind, width=w, height=h, mean_k=rng.randint(8, 50))
    elif kind == "mls":
        w, h = _draw_size(rng, 640, 2048)
        if rng.random() < 0.5:
            return dict(kind=kind, width=w, height=h, order=rng.choice([0, 1]), window=rng.randint(10, 30),
                        sigma=rng.choice([0.5, 0.6, 0.8]), radius=0.0, iterations=rng.randint(1, 3))
        r = rng.uniform(1.5, 2.5)
        return dict(kind=kind, width=w, height=h, order=2, window=rng.randint(5, 9), sigma=r / math.sqrt(2.0),
                    radius=r, iterations=1)
    elif kind == "metric_gaussian":
        w, h = _draw_size(rng, 640, 2448)
        return dict(kind=kind, width=w, height=h, sigma=rng.choice([0.3, 0.4, 0.5]))
    else:
        w, h = _draw_size(rng, 640, 2448)
        return dict(kind=kind, width=w, height=h, poses=rng.randint(1, 4))
    return dict(kind=kind, width=w, height=h)


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _spec(encoding, width, height, seed, hdr=False):
    """A rendered scene: the library's own seeded scenes at the case's size."""
    if encoding == "gray":
        return synth.config0(seed, width, height)
    if encoding == "hier":
        return synth.config1(seed, width, height)
    s = synth.ref_heterodyne(seed, width, height)
    if hdr:
        s.A, s.B = (110, 170), (70, 120)  # bright enough that crests saturate at 255
    return s


def _decode_cfg(spec, hdr=False):
    kw = spec.decode_kwargs()
    if hdr:
        kw.update(enable_hdr=True, hdr_saturation_gray=255.0 if spec.bit_depth == 8 else 3000.0,
                  hdr_min_amplitude=2.0 if spec.bit_depth == 8 else 32.0)
    return api.decode_config(**kw)


def _frames(spec, cam):
    return torch.from_numpy(spec.render(cam)).cuda()


def _context(spec):
    ctx = api.Context(torch.cuda.current_device())
    ctx.set_calibration(spec.rig.as_dict(), True)
    return ctx


def _recon_cfg(case):
    kw = dict(use_px_gaussian=0, use_ror=0, use_sor=1, sor_mean_k=case["mean_k"], sor_std_mul=1.0)
    if case["smooth"]:
        kw.update(use_mls=1, mls_window_size=7, mls_spatial_sigma=2.0 / math.sqrt(2.0), mls_polynomial_order=2,
                  mls_max_radius=2.0, mls_iterations=1, use_metric_gaussian=1, metric_gaussian_sigma=0.5)
    return api.recon_config(**kw)


def _decoded_pair(spec):
    """Orders (int32) and residuals (float32) of both cameras, decoded with plain torch."""
    out = []
    for cam in (0, 1):
        k, r, ok, _ = _decode64(_frames(spec, cam), spec)
        out.append((torch.where(ok, k, 0).to(torch.int32), torch.where(ok, r, 0.0).to(torch.float32)))
    return out


def _cloud(ctx, seed):
    """An organised cloud as the reprojection leaves it, every point on its pixel's
    ray: a plane with smooth bumps and two boxes in front, depth mixed across the
    box edges (the post-smooth's flying pixels), occlusion gaps beside the boxes,
    an invalid rim, dropped pixels, measurement noise and a few gross outliers."""
    g = torch.Generator(device="cuda")
    g.manual_seed(7919 * seed + 11)
    H, W = ctx.rect_h, ctx.rect_w
    cx, cy, f = -ctx.Q[0, 3], -ctx.Q[1, 3], ctx.Q[2, 3]
    q32, q33 = ctx.Q[3, 2], ctx.Q[3, 3]
    dev = "cuda"

    def uni(n, lo, hi):
        return (torch.rand(n, generator=g, device=dev, dtype=torch.float64) * (hi - lo) + lo).tolist()

    x = (torch.arange(W, device=dev, dtype=torch.float64) - cx) * (PLANE_Z / f)
    y = (torch.arange(H, device=dev, dtype=torch.float64) - cy) * (PLANE_Z / f)
    z = torch.full((H, W), PLANE_Z, device=dev, dtype=torch.float64)
    for bx, by, a, s in zip(uni(20, -400, 400), uni(20, -330, 330), uni(20, 5, 40), uni(20, 20, 150)):
        z -= a * torch.exp(-0.5 * (((y - by) / s) ** 2)[:, None] - 0.5 * (((x - bx) / s) ** 2)[None, :])
    gap = torch.zeros((H, W), device=dev, dtype=torch.bool)
    for b0, b1, bw, bh, bz in zip(uni(2, -300, 100), uni(2, -250, 50), uni(2, 120, 250), uni(2, 120, 250),
                                  uni(2, 60, 120)):
        iny = ((y >= b1) & (y < b1 + bh))[:, None]
        z = torch.where(iny & ((x >= b0) & (x < b0 + bw))[None, :], PLANE_Z - bz, z)
        shadow = 100.0 * bz / (PLANE_Z - bz)  # the projector's shadow beside the box
        gap |= iny & ((x >= b0 - shadow) & (x < b0))[None, :]
    d = (ctx.Q[2, 3] / z - q33) / q32
    p = torch.nn.functional.pad(d[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
    d = sum(wa * wb * p[a:a + H, b:b + W] for a, wa in enumerate((0.25, 0.5, 0.25))
            for b, wb in enumerate((0.25, 0.5, 0.25)))
    z = ctx.Q[2, 3] / (q32 * d + q33)
    z = z + 0.03 * torch.randn((H, W), generator=g, device=dev, dtype=torch.float64)
    u = torch.rand((H, W), generator=g, device=dev)
    z = torch.where(u < 0.0003, z - 15.0 - 40.0 * torch.rand((H, W), generator=g, device=dev), z)
    mask = ~gap & (u < 0.995)
    rim = max(2, W // 60)
    mask[:, :rim] = False
    mask[:, W - rim:] = False
    mask[:2] = False
    mask[H - 2:] = False
    col = torch.arange(W, device=dev, dtype=torch.float64)[None, :] - cx
    row = torch.arange(H, device=dev, dtype=torch.float64)[:, None] - cy
    xyz = torch.stack([col * z / f, row * z / f, z], dim=-1)
    xyz = torch.where(mask[..., None], xyz, 0.0).to(torch.float32)
    return xyz.contiguous(), mask.to(torch.uint8).contiguous()


def _cloud_context(case):
    return _context(synth.config1(1, case["width"], case["height"]))


def _undistort(rig, cam, W, H):
    """Normalised ray of every source pixel (the distortion undone by fixed-point steps)."""
    K, D = np.asarray(rig.K[cam], float), np.asarray(rig.D[cam], float)
    xd = ((torch.arange(W, device="cuda", dtype=torch.float64) - K[0, 2]) / K[0, 0])[None, :].expand(H, W)
    yd = ((torch.arange(H, device="cuda", dtype=torch.float64) - K[1, 2]) / K[1, 1])[:, None].expand(H, W)
    x, y = xd, yd
    for _ in range(12):
        r2 = x * x + y * y
        s = 1.0 + r2 * (D[0] + r2 * D[1])
        x, y = xd / s, yd / s
    return x, y


def _plane_view(ctx, spec, seed):
    """One pose of a planar target: decoded phase of both cameras (exact phase plus
    decoding noise), match columns from the geometry, the plane as (n, d)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rig = spec.rig
    W, H = rig.width, rig.height
    B = -float(rig.t[0])
    n, pd = np.asarray(spec.plane_n, float), float(spec.plane_d)
    orders, residuals = [], []
    for cam in (0, 1):
        x, y = _undistort(rig, cam, W, H)
        z = (pd - n[0] * B * cam) / (n[0] * x + n[1] * y + n[2])
        X = x * z + B * cam
        u = spec.proj_f * (X - spec.proj_center[0]) / z + (spec.proj_width - 1) / 2
        v = spec.proj_f * (y * z - spec.proj_center[1]) / z + (spec.proj_height - 1) / 2
        phase = TWO_PI * spec.freq[-1] * u / spec.proj_width
        phase = phase + 0.01 * torch.randn(phase.shape, generator=g, device="cuda", dtype=torch.float64)
        k = torch.floor(phase / TWO_PI + 0.5)
        ok = (u >= 0) & (u < spec.proj_width) & (v >= 0) & (v < spec.proj_height) & (k >= 1)
        ok &= torch.rand(phase.shape, generator=g, device="cuda") < 0.999
        orders.append(torch.where(ok, k, 0.0).to(torch.int32).contiguous())
        residuals.append(torch.where(ok, phase - TWO_PI * k, 0.0).to(torch.float32).contiguous())
    rh, rw = ctx.rect_h, ctx.rect_w
    Q = ctx.Q
    ray = [torch.arange(rw, device="cuda", dtype=torch.float64)[None, :] + Q[0, 3],
           torch.arange(rh, device="cuda", dtype=torch.float64)[:, None] + Q[1, 3]]
    w = (n[0] * ray[0] + n[1] * ray[1] + n[2] * Q[2, 3]) / pd  # the point is ray / w
    d = (w - Q[3, 3]) / Q[3, 2]
    col = torch.arange(rw, device="cuda", dtype=torch.float64)[None, :] - d
    best = torch.where((col >= 2) & (col < rw - 2) & (w > 0), torch.round(col), -1.0).to(torch.int32).contiguous()
    return orders, residuals, best, (n[0], n[1], n[2], -pd)


def _diff_inputs(case, seed):
    spec = synth.config1(1, case["width"], case["height"])
    ctx = _context(spec)
    views = []
    for p in range(case["poses"]):
        s = synth.pose_plane(3 + seed, case["width"], case["height"], p)
        views.append(_plane_view(ctx, s, 1000 * seed + p))
    theta = diff.nominal(ctx)
    # the refinement's start: baseline +0.5 %, cx0 +3 px, k1_0 +0.02
    theta[12] *= 1.005
    theta[2] += 3.0
    theta[4] += 0.02
    return spec, ctx, views, theta


# --------------------------------------------------------------------------
# prepare / run
# --------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "pair":
        spec = _spec(case["encoding"], case["width"], case["height"], seed + 1)
        ctx = _context(spec)
        out = (torch.empty((ctx.rect_h, ctx.rect_w, 3), dtype=torch.float32, device="cuda"),
               torch.empty((ctx.rect_h, ctx.rect_w), dtype=torch.uint8, device="cuda"),
               torch.empty((ctx.rect_h, ctx.rect_w), dtype=torch.float32, device="cuda"))
        return dict(kind=kind, ctx=ctx, dcfg=_decode_cfg(spec), rcfg=_recon_cfg(case), left=_frames(spec, 0),
                    right=_frames(spec, 1), out=out)
    if kind == "decode":
        spec = _spec(case["encoding"], case["width"], case["height"], seed + 1, case["hdr"])
        return dict(kind=kind, ctx=api.Context(torch.cuda.current_device()), dcfg=_decode_cfg(spec, case["hdr"]),
                    frames=_frames(spec, 0))
    if kind in ("rectify_match", "reconstructor"):
        spec = _spec("hier", case["width"], case["height"], seed + 1)
        left, right = _decoded_pair(spec)
        if kind == "rectify_match":
            return dict(kind=kind, ctx=_context(spec), left=left, right=right, pha_f=spec.pha_f)
        cls = api.JSLAB_PhaseEpipolarReconstructor_V2
        rec = cls(cls.Config(radius_search=case["radius"]))
        d = spec.rig.as_dict()
        rec.setCalibrationParams(api.JSLAB_StereoCalibParams_V1(d["K"], d["D"], d["R"], d["t"],
                                                                (d["width"], d["height"])))
        return dict(kind=kind, rec=rec, left=api.DecodedPhase(*left, None, None, True),
                    right=api.DecodedPhase(*right, None, None, True), pha_f=spec.pha_f)
    if kind in ("sor", "mls", "metric_gaussian"):
        ctx = _cloud_context(case)
        xyz, mask = _cloud(ctx, seed)
        return dict(kind=kind, ctx=ctx, xyz=xyz, mask=mask, case=dict(case))
    _, ctx, views, theta = _diff_inputs(case, seed)
    return dict(kind=kind, ctx=ctx, theta=theta, views=[diff.View(o, r, b, p) for o, r, b, p in views])


def run(state):
    kind = state["kind"]
    if kind == "pair":
        return api.reconstruct_pair(state["ctx"], state["dcfg"], state["rcfg"], state["left"], state["right"],
                                    out=state["out"])
    if kind == "decode":
        return api.decode(state["ctx"], state["dcfg"], state["frames"])
    if kind == "rectify_match":
        return api.rectify_match(state["ctx"], state["left"], state["right"], state["pha_f"])
    if kind == "reconstructor":
        rec = state["rec"]
        rec.setData(state["left"], state["right"], pha_f=state["pha_f"])
        return rec.startCalculate()
    c = state["case"] if "case" in state else None
    if kind == "sor":
        return api.filter_sor(state["ctx"], state["xyz"], state["mask"], c["mean_k"], 1.0, want_mean_dist=True)
    if kind == "mls":
        return api.filter_mls(state["ctx"], state["xyz"], state["mask"], c["window"], c["sigma"], c["order"],
                              c["radius"], c["iterations"])
    if kind == "metric_gaussian":
        return api.filter_metric_gaussian(state["ctx"], state["xyz"], state["mask"], c["sigma"])
    return diff.backward(state["ctx"], state["theta"], state["views"], 1.0, 1.0, 5000.0)


# --------------------------------------------------------------------------
# work
# --------------------------------------------------------------------------
_FORMAT = {"gray": (10, 1, 1, 4), "hier": (12, 2, 3, 12), "hetero": (24, 1, 3, 24)}  # frames, bytes, freqs, steps


def _decode_flops(encoding):
    """Per pixel: three sums per phase sample, a 3 x 3 blur of three sums, an arctangent and the unwrapping."""
    _, _, nf, steps = _FORMAT[encoding]
    return 5 * steps + nf * (54 + 30) + 20


def _window(case, radius):
    """Pixels of a disk of the given radius in millimetres on the background plane."""
    f = 2400.0 * case["width"] / 2448.0
    return max(1.0, math.pi * (radius * f / PLANE_Z) ** 2)


def work(case):
    kind, n = case["kind"], float(case["width"]) * case["height"]
    if kind == "pair":
        F, es, _, _ = _FORMAT[case["encoding"]]
        flops = 2 * n * _decode_flops(case["encoding"]) + n * (150 + 100 + 8 * 2 * case["mean_k"])
        if case["smooth"]:
            flops += n * (56 * _window(case, 2.0) + 16 * _window(case, 1.5))
        return {"bytes": 2 * n * F * es + n * (13 + 4), "flops": flops}
    if kind == "decode":
        F, es, _, _ = _FORMAT[case["encoding"]]
        return {"bytes": n * F * es + n * 13, "flops": n * _decode_flops(case["encoding"])}
    if kind == "rectify_match":
        return {"bytes": 2 * n * 8 + n * 4, "flops": n * 150}
    if kind == "reconstructor":
        return {"bytes": 2 * n * 8 + n * 13, "flops": n * (150 + 100 + 9 * 10 + 11 * 8)}
    if kind == "sor":
        return {"bytes": n * (13 + 5), "flops": n * 8 * 2 * case["mean_k"]}
    if kind == "mls":
        r = case["radius"] if case["radius"] > 0 else 3 * case["sigma"]
        per = 56 if case["order"] == 2 else 20
        return {"bytes": n * (13 + 12), "flops": n * case["iterations"] * per * _window(case, r)}
    if kind == "metric_gaussian":
        return {"bytes": n * (13 + 12), "flops": n * 16 * _window(case, 3 * case["sigma"])}
    v = case["poses"]
    return {"bytes": v * n * (2 * 8 + 4), "flops": v * n * (4 * 120 + 136 * 2 + 64)}


# --------------------------------------------------------------------------
# exact: the same outputs in 64 bits, plain torch
# --------------------------------------------------------------------------
def _blur3(a, k):
    """3 x 3 blur with the separable kernel k and replicated borders."""
    H, W = a.shape
    p = torch.nn.functional.pad(a[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
    return sum(k[i] * k[j] * p[i:i + H, j:j + W] for i in range(3) for j in range(3))


def _wide(frames):
    """Samples as float64 (u16 samples go through int32)."""
    if frames.dtype == torch.uint16:
        return (frames.view(torch.int16).to(torch.int32) & 0xffff).to(torch.float64)
    return frames.to(torch.float64)


def _decode64(frames, spec, hdr=False):
    """(order, residual, valid, modulation) of a fringe stack."""
    kw = spec.decode_kwargs()
    t = math.exp(-0.5 / kw["preblur_sigma"] ** 2)
    kb = [t / (1 + 2 * t), 1 / (1 + 2 * t), t / (1 + 2 * t)]
    H, W = frames.shape[1:]
    ok = torch.ones((H, W), dtype=torch.bool, device=frames.device)
    wraps, mod0, f0 = [], None, 0
    sat = 255.0 if spec.bit_depth == 8 else 3000.0
    min_amp = 2.0 if spec.bit_depth == 8 else 32.0
    for i in range(spec.n_freq):
        N = spec.shift_num[i]
        I = _wide(frames[f0:f0 + N])
        f0 += N
        ang = TWO_PI * torch.arange(N, device=I.device, dtype=torch.float64) / N
        sn, cs = torch.sin(ang), torch.cos(ang)
        if hdr:
            m = ((I >= 0) & (I < sat)).to(torch.float64)
            cnt = m.sum(0)
            basis = [torch.ones_like(cs), cs, -sn]
            G = torch.stack([torch.stack([torch.einsum("n,nhw->hw", a * b, m) for b in basis], -1) for a in basis], -2)
            rhs = torch.stack([torch.einsum("n,nhw->hw", a, m * I) for a in basis], -1)
            fit = cnt >= 3
            G = torch.where(fit[..., None, None], G, torch.eye(3, dtype=torch.float64, device=I.device))
            det = (G[..., 0, 0] * (G[..., 1, 1] * G[..., 2, 2] - G[..., 1, 2] ** 2)
                   - G[..., 0, 1] * (G[..., 0, 1] * G[..., 2, 2] - G[..., 1, 2] * G[..., 0, 2])
                   + G[..., 0, 2] * (G[..., 0, 1] * G[..., 1, 2] - G[..., 1, 1] * G[..., 0, 2]))
            fit &= det.abs() > 1e-6 * cnt ** 3
            A, C, S = _solve3(G, rhs, det)
            ok &= fit & (torch.hypot(C, S) > min_amp) & (A > 1e-3)
            S, C, M = S * N / 2, C * N / 2, A * N
        else:
            S = _blur3(-torch.einsum("n,nhw->hw", sn, I), kb)
            C = _blur3(torch.einsum("n,nhw->hw", cs, I), kb)
            M = _blur3(I.sum(0), kb)
        wraps.append(torch.atan2(S, C))
        nm = torch.where(M > 1e-3 * N, 2 * torch.hypot(S, C) / M, 0.0)
        mod0 = nm if i == 0 else mod0
        ok &= ~(nm < kw["modulation_threshold"])
    rnd = lambda v: torch.trunc(v + torch.copysign(torch.full_like(v, 0.5), v))
    if spec.encoding == synth.ENC_HETERODYNE3:
        F0, F1, F2 = (float(v) for v in spec.freq[:3])
        f12, f23 = abs(F0 - F1), abs(F1 - F2)
        w0, w1, w2 = wraps
        p12 = torch.where(w0 > w1, w0 - w1, w0 - w1 + TWO_PI)
        a, b = (w1, w2) if F1 > F2 else (w2, w1)
        p23 = torch.where(a > b, a - b, a - b + TWO_PI)
        p123 = torch.where(p12 > p23, p12 - p23, p12 - p23 + TWO_PI)
        u12 = p12 + TWO_PI * rnd((p123 * f12 - p12) / TWO_PI)
        k = rnd((u12 * F0 / f12 - w0) / TWO_PI)
        u23 = p23 + TWO_PI * rnd((p123 * f23 - p23) / TWO_PI)
        u1 = w1 + TWO_PI * rnd((u23 * F1 / f23 - w1) / TWO_PI)
        u2 = w2 + TWO_PI * rnd((u23 * F2 / f23 - w2) / TWO_PI)
        r = (w0 + (u1 * F0 / F1 - TWO_PI * k) + (u2 * F0 / F2 - TWO_PI * k)) / 3.0
    elif spec.encoding == synth.ENC_HIERARCHICAL:
        k = torch.zeros_like(wraps[0])
        for i in range(1, spec.n_freq):
            q = spec.freq[i] / spec.freq[i - 1]
            k = q * k + rnd((q * (wraps[i - 1] + math.pi) - (wraps[i] + math.pi)) / TWO_PI)
        r = wraps[-1]
    else:
        N, w = spec.shift_num[0], wraps[0]
        I = _wide(frames)
        mean = I[:N].sum(0)
        bits = [(N * I[N + b] > mean).to(torch.int64) for b in range(spec.gray_bits + 1)]
        v = torch.zeros_like(bits[0])
        last = torch.zeros_like(bits[0])
        for b in bits[:spec.gray_bits]:
            last = last ^ b
            v = 2 * v + last
        k2 = (2 * v + (last ^ bits[-1]) + 1) // 2
        k = torch.where(w <= -math.pi / 2, k2, torch.where(w >= math.pi / 2, k2 - 1, v)).to(torch.float64)
        r = w
    return k, r, ok, mod0


def _solve3(G, rhs, det):
    """Symmetric 3 x 3 systems by cofactors."""
    g = lambda i, j: G[..., i, j]
    c = [g(1, 1) * g(2, 2) - g(1, 2) ** 2, g(0, 2) * g(1, 2) - g(0, 1) * g(2, 2), g(0, 1) * g(1, 2) - g(0, 2) * g(1, 1),
         g(0, 0) * g(2, 2) - g(0, 2) ** 2, g(0, 1) * g(0, 2) - g(0, 0) * g(1, 2), g(0, 0) * g(1, 1) - g(0, 1) ** 2]
    b = [rhs[..., i] for i in range(3)]
    return [(c[0] * b[0] + c[1] * b[1] + c[2] * b[2]) / det, (c[1] * b[0] + c[3] * b[1] + c[4] * b[2]) / det,
            (c[2] * b[0] + c[4] * b[1] + c[5] * b[2]) / det]


def _remap(ctx, rig, cam, order, phase):
    """Rectified (order, phase): nearest order, bilinear phase on 1/32-pixel positions, 0 outside."""
    H, W = order.shape
    K, D = np.asarray(rig.K[cam], float), np.asarray(rig.D[cam], float)
    P, R = (ctx.P1, ctx.R1) if cam == 0 else (ctx.P2, ctx.R2)
    ir = np.linalg.inv(P[:, :3] @ R)
    j = torch.arange(ctx.rect_w, device="cuda", dtype=torch.float64)[None, :]
    i = torch.arange(ctx.rect_h, device="cuda", dtype=torch.float64)[:, None]
    ww = ir[2, 0] * j + ir[2, 1] * i + ir[2, 2]
    x = (ir[0, 0] * j + ir[0, 1] * i + ir[0, 2]) / ww
    y = (ir[1, 0] * j + ir[1, 1] * i + ir[1, 2]) / ww
    r2 = x * x + y * y
    kr = 1 + ((D[4] * r2 + D[1]) * r2 + D[0]) * r2
    mx = (K[0, 0] * (x * kr + D[2] * 2 * x * y + D[3] * (r2 + 2 * x * x)) + K[0, 2]).to(torch.float32)
    my = (K[1, 1] * (y * kr + D[2] * (r2 + 2 * y * y) + D[3] * 2 * x * y) + K[1, 2]).to(torch.float32)

    def tap(a, xx, yy):
        inside = (xx >= 0) & (yy >= 0) & (xx < W) & (yy < H)
        return torch.where(inside, a[yy.clamp(0, H - 1), xx.clamp(0, W - 1)], 0)

    ro = tap(order, torch.round(mx).to(torch.int64), torch.round(my).to(torch.int64))
    sx, sy = torch.round(mx * 32).to(torch.int64), torch.round(my * 32).to(torch.int64)
    x0, y0 = sx >> 5, sy >> 5
    fx, fy = (sx & 31).to(torch.float64) / 32, (sy & 31).to(torch.float64) / 32
    ph = ((1 - fy) * ((1 - fx) * tap(phase, x0, y0) + fx * tap(phase, x0 + 1, y0))
          + fy * ((1 - fx) * tap(phase, x0, y0 + 1) + fx * tap(phase, x0 + 1, y0 + 1)))
    return ro, ph


def _match64(ctx, rig, left, right, pha_f, grad=1.0):
    """Disparity of two decoded cameras: post-smooth, remap, first column of least phase difference."""
    rects = []
    for cam, (k, r) in enumerate((left, right)):
        ph = _blur3(TWO_PI * k.to(torch.float64) + r.to(torch.float64), (0.25, 0.5, 0.25))
        rects.append(_remap(ctx, rig, cam, k, ph))
    (lo, lp), (ro, rp) = rects
    H, W = lo.shape
    disp = torch.zeros((H, W), dtype=torch.float64, device=lp.device)
    step = max(1, int(2.5e8 // (W * W)))
    col = torch.arange(W, device=lp.device)[None, :]
    for a in range(0, H, step):
        s = slice(a, min(H, a + step))
        cost = (rp[s][:, None, :] - lp[s][:, :, None]).abs()
        cost.masked_fill_(ro[s][:, None, :] != lo[s][:, :, None], 1e9)
        best, bj = cost.min(dim=2)
        bj = torch.where(cost.gather(2, bj[..., None])[..., 0] < 1e9, bj, 0)
        ok = (lo[s] >= 1) & (lo[s] <= pha_f) & (best < grad) & (bj >= 2) & (bj < W - 1)
        b = bj.clamp(1, W - 2)
        c0, c1, c2 = (rp[s].gather(1, b + o) - lp[s] for o in (-1, 0, 1))
        den = 2 * (c0 - c1) * (c1 - c2)
        delta = torch.where(den.abs() > 1e-9, c1 * (c0 - c2) / den, 0.0)
        disp[s] = torch.where(ok, (col - bj).to(torch.float64) - delta, 0.0)
        del cost
    return disp


def _pad(a, r, value):
    """a (H, W[, C]) with r rows and columns of `value` around it."""
    pads = (0, 0) * (a.dim() - 2) + (r, r, r, r)
    return torch.nn.functional.pad(a, pads, value=value)


def _reconstruct64(ctx, disp, min_depth=0.0, max_depth=1000.0, radius=0.7, min_nb=10, window=10):
    """Median, reprojection, 3 x 3 point Gaussian, radius outlier filter (the class's defaults)."""
    H, W = disp.shape
    p = torch.nn.functional.pad(disp[None, None], (2, 2, 2, 2), mode="replicate")[0, 0]
    med = torch.empty_like(disp)
    for a in range(0, H, 256):
        b = min(H, a + 256)
        med[a:b] = torch.stack([p[a + i:b + i, j:j + W] for i in range(5) for j in range(5)]).median(dim=0).values
    Q = ctx.Q
    w = Q[3, 2] * med + Q[3, 3]
    x = (torch.arange(W, device=disp.device, dtype=torch.float64)[None, :] + Q[0, 3]) / w
    y = (torch.arange(H, device=disp.device, dtype=torch.float64)[:, None] + Q[1, 3]) / w
    z = Q[2, 3] / w
    m = (med.abs() >= 1e-5) & (z > min_depth) & (z < max_depth)
    P = torch.where(m[..., None], torch.stack([x, y, z], -1), 0.0)
    k1 = 1.0 / (1.0 + 2.0 * math.exp(-0.5 / 0.49))
    kern = ((1 - k1) / 2, k1, (1 - k1) / 2)
    Pp, mp = _pad(P, 1, 0.0), _pad(m, 1, False)
    acc, cnt = torch.zeros_like(P), torch.zeros_like(disp)
    for i in range(3):
        for j in range(3):
            q = Pp[i:i + H, j:j + W]
            use = mp[i:i + H, j:j + W] & ((q[..., 0] - P[..., 0]).abs() < 3.0)
            wt = torch.where(use, kern[i] * kern[j], 0.0)
            acc += wt[..., None] * q
            cnt += wt
    inner = torch.zeros_like(m)
    inner[1:H - 1, 1:W - 1] = True
    G = torch.where((m & inner & (cnt > 0.8))[..., None], acc / cnt.clamp_min(1e-300)[..., None], 0.0)
    hw = window // 2
    Gp = _pad(torch.where(m[..., None], G, math.nan), hw, math.nan)
    nb = torch.zeros_like(cnt)
    for i in range(2 * hw + 1):
        for j in range(2 * hw + 1):
            if i != hw or j != hw:
                nb += ((Gp[i:i + H, j:j + W] - G) ** 2).sum(-1) <= float(np.float32(radius)) ** 2
    return torch.where((m & (nb >= min_nb))[..., None], G, 0.0)


def _reach(ctx, xyz, mask, radius, limit):
    """Window half-size that holds every point within `radius` of another (points lie on their pixel rays)."""
    z = float(xyz[..., 2][mask > 0].min()) - radius
    tan = max(ctx.rect_w, ctx.rect_h) / abs(float(ctx.Q[2, 3]))
    return min(limit, int(abs(float(ctx.Q[2, 3])) * radius * (1 + tan) / z) + 2)


def _normal(C):
    """Unit eigenvector of the smallest eigenvalue of symmetric 3 x 3 matrices (six entries xx xy xz yy yz zz)."""
    a, b, c, d, e, f = C
    q = (a + d + f) / 3
    p = torch.sqrt(((a - q) ** 2 + (d - q) ** 2 + (f - q) ** 2 + 2 * (b * b + c * c + e * e)) / 6).clamp_min(1e-150)
    A, D, F = (a - q) / p, (d - q) / p, (f - q) / p
    B, Cc, E = b / p, c / p, e / p
    det = A * (D * F - E * E) - B * (B * F - E * Cc) + Cc * (B * E - D * Cc)
    ev = q + 2 * p * torch.cos(torch.acos((det / 2).clamp(-1, 1)) / 3 + TWO_PI / 3)
    r0, r1, r2 = torch.stack([a - ev, b, c], -1), torch.stack([b, d - ev, e], -1), torch.stack([c, e, f - ev], -1)
    cand = torch.stack([torch.linalg.cross(r0, r1), torch.linalg.cross(r0, r2), torch.linalg.cross(r1, r2)], -2)
    n2 = (cand ** 2).sum(-1)
    pick = n2.argmax(-1)
    v = cand.gather(-2, pick[..., None, None].expand(*pick.shape, 1, 3))[..., 0, :]
    return v / v.norm(dim=-1, keepdim=True).clamp_min(1e-300)


def _mls_pass(P, mask, R, hw, sigma, order, r2):
    """One MLS pass over the valid pixels; neighbours up to R pixels away (all within the window hw)."""
    H, W = mask.shape
    R = min(R, hw)
    Pn = _pad(torch.where(mask[..., None], P, math.nan), R, math.nan)
    ks = -0.5 / float(np.float32(sigma)) ** 2

    def visit():
        for i in range(2 * R + 1):
            for j in range(2 * R + 1):
                d = Pn[i:i + H, j:j + W] - P
                d2 = (d * d).sum(-1)
                use = d2 <= r2
                yield (torch.where(use[..., None], d, 0.0), torch.where(use, torch.exp(ks * d2), 0.0), use)

    ws, nv = torch.zeros((H, W), dtype=torch.float64, device=P.device), torch.zeros((H, W), device=P.device)
    s1 = torch.zeros_like(P)
    s2 = [torch.zeros_like(ws) for _ in range(6)]
    for d, w, use in visit():
        x, y, z = d.unbind(-1)
        ws += w
        nv += use
        s1 += w[..., None] * d
        for t, v in zip(s2, (x * x, x * y, x * z, y * y, y * z, z * z)):
            t += w * v
    live = mask & (nv >= 3) & (ws >= 1e-12)
    c = s1 / ws.clamp_min(1e-300)[..., None]
    cx, cy, cz = c.unbind(-1)
    C = [t - ws * v for t, v in zip(s2, (cx * cx, cx * cy, cx * cz, cy * cy, cy * cz, cz * cz))]
    n = _normal(C)
    axis = torch.nn.functional.one_hot(n.abs().argmin(-1), 3).to(torch.float64)
    t1 = axis - (axis * n).sum(-1, keepdim=True) * n
    t1 = t1 / t1.norm(dim=-1, keepdim=True).clamp_min(1e-300)
    t2 = torch.linalg.cross(n, t1)
    need = {0: 3, 1: 5, 2: 8}[order]
    cur = torch.where(nv >= need, order, 0)
    h = math.sqrt(r2)
    u0, v0 = -(c * t1).sum(-1) / h, -(c * t2).sum(-1) / h
    f0 = -(c * n).sum(-1)
    fit = torch.zeros_like(ws)  # height of the fitted surface at the query's (u0, v0)
    M = torch.stack([torch.stack([C[0], C[1], C[2]], -1), torch.stack([C[1], C[3], C[4]], -1),
                     torch.stack([C[2], C[4], C[5]], -1)], -2)
    frame = torch.stack([t1 / h, t2 / h, n], -2)
    m = frame @ M @ frame.transpose(-1, -2)
    if order >= 1:
        det = m[..., 0, 0] * m[..., 1, 1] - m[..., 0, 1] ** 2
        a1 = (m[..., 1, 1] * m[..., 0, 2] - m[..., 0, 1] * m[..., 1, 2]) / det
        a2 = (m[..., 0, 0] * m[..., 1, 2] - m[..., 0, 1] * m[..., 0, 2]) / det
        fit = torch.where((cur >= 1) & (det > 1e-24), a1 * u0 + a2 * v0, 0.0)
    if order == 2:
        mom = {e: torch.zeros_like(ws) for e in ((3, 0), (2, 1), (1, 2), (0, 3), (4, 0), (3, 1), (2, 2), (1, 3), (0, 4))}
        rhs = [torch.zeros_like(ws) for _ in range(3)]
        for d, w, _ in visit():
            e = d - c
            u, v, f = (e * t1).sum(-1) / h, (e * t2).sum(-1) / h, (e * n).sum(-1)
            for (a, b), t in mom.items():
                t += w * u ** a * v ** b
            rhs[0] += w * f * u * u
            rhs[1] += w * f * u * v
            rhs[2] += w * f * v * v
        mom.update({(0, 0): ws, (1, 0): torch.zeros_like(ws), (0, 1): torch.zeros_like(ws), (2, 0): m[..., 0, 0],
                    (1, 1): m[..., 0, 1], (0, 2): m[..., 1, 1]})
        ex = [(0, 0), (1, 0), (0, 1), (2, 0), (1, 1), (0, 2)]
        sel = (cur == 2) & live
        b = torch.stack([torch.zeros_like(ws), m[..., 0, 2], m[..., 1, 2], *rhs], -1)[sel]
        A = torch.stack([torch.stack([mom[(p[0] + q[0], p[1] + q[1])][sel] for q in ex], -1) for p in ex], -2)
        x = torch.zeros_like(b)
        good = torch.zeros(b.shape[0], dtype=torch.bool, device=b.device)
        for s in range(0, b.shape[0], 400000):
            L, info = torch.linalg.cholesky_ex(A[s:s + 400000])
            x[s:s + 400000] = torch.cholesky_solve(b[s:s + 400000, :, None], L)[..., 0]
            good[s:s + 400000] = info == 0
        uu, vv = u0[sel], v0[sel]
        f2 = x[:, 0] + x[:, 1] * uu + x[:, 2] * vv + x[:, 3] * uu * uu + x[:, 4] * uu * vv + x[:, 5] * vv * vv
        fit[sel] = torch.where(good, f2, fit[sel])
    moved = P + (fit - f0)[..., None] * n
    return torch.where(live[..., None], moved, P)


def _mls64(ctx, xyz, mask, case):
    s = np.float32(case["sigma"])
    r2 = float(np.float32(case["radius"]) ** 2) if case["radius"] > 0 else float(np.float32(9.0) * s * s)
    R = _reach(ctx, xyz, mask, math.sqrt(r2), case["window"])
    P, m = xyz.to(torch.float64), mask > 0
    for _ in range(case["iterations"]):
        P = _mls_pass(P, m, R, case["window"], case["sigma"], case["order"], r2)
    return P


def _metric_gaussian64(ctx, xyz, mask, sigma):
    H, W = mask.shape
    P, m = xyz.to(torch.float64), mask > 0
    r = 3.0 * sigma
    R = _reach(ctx, xyz, mask, r, 64)
    Pn = _pad(torch.where(m[..., None], P, math.nan), R, math.nan)
    r2 = float(np.float32(r) * np.float32(r))
    acc, cnt = torch.zeros_like(P), torch.zeros((H, W), dtype=torch.float64, device=P.device)
    for i in range(2 * R + 1):
        for j in range(2 * R + 1):
            d = Pn[i:i + H, j:j + W] - P
            d2 = (d * d).sum(-1)
            w = torch.where(d2 <= r2, torch.exp(-d2 / (2 * sigma * sigma)), 0.0)
            acc += torch.where(d2 <= r2, w, 0.0)[..., None] * torch.nan_to_num(d)
            cnt += w
    return torch.where(m[..., None], P + acc / cnt.clamp_min(1e-300)[..., None], P)


def _sor64(ctx, xyz, mask, k):
    """Mean distance of every valid point to its k nearest: a pixel window where
    it provably holds them (points lie on their pixel rays), else all points."""
    H, W = mask.shape
    P, m = xyz.to(torch.float64), mask > 0
    R = 9
    Pn = _pad(torch.where(m[..., None], P, math.inf), R, math.inf)
    md, kth = torch.zeros((H, W), dtype=torch.float64, device=P.device), torch.zeros_like(P[..., 0])
    for a in range(0, H, 32):
        b = min(H, a + 32)
        d2 = torch.stack([((Pn[a + i:b + i, j:j + W] - P[a:b]) ** 2).sum(-1) for i in range(2 * R + 1)
                          for j in range(2 * R + 1)], -1)
        v = torch.nan_to_num(d2, nan=math.inf).topk(k + 1, dim=-1, largest=False).values.sqrt()
        md[a:b] = v.sum(-1) / k
        kth[a:b] = v.amax(-1)
    f = abs(float(ctx.Q[2, 3]))
    tan = (P[..., 0].abs() + P[..., 1].abs()) / P[..., 2].clamp_min(1e-6)
    sure = (P[..., 2] > kth) & (f * kth * (1 + tan) / (P[..., 2] - kth) < R)
    rest = (m & ~sure).nonzero()
    pts = P[m]
    for a in range(0, rest.shape[0], 256):
        ij = rest[a:a + 256]
        q = P[ij[:, 0], ij[:, 1]]
        d = torch.cdist(q, pts, compute_mode="donot_use_mm_for_euclid_dist")
        md[ij[:, 0], ij[:, 1]] = d.topk(k + 1, dim=-1, largest=False).values.sum(-1) / k
    return torch.where(m, md, 0.0)


def _diff64(spec, ctx, views, theta, zmin=1.0, zmax=5000.0):
    """Loss, points, gradient and J^T J of the point-to-plane distances, by forward-mode differentiation."""
    rh, rw = ctx.rect_h, ctx.rect_w
    H, W = spec.rig.height, spec.rig.width
    Q = ctx.Q
    ir = [torch.tensor(np.linalg.inv(P[:, :3] @ R), device="cuda")
          for P, R in ((ctx.P1, ctx.R1), (ctx.P2, ctx.R2))]
    B0 = float(np.linalg.norm(spec.rig.t))
    Tx0 = -1.0 / Q[3, 2]
    dcx = Q[3, 3] * Tx0
    j = torch.arange(rw, device="cuda", dtype=torch.float64)[None, :].expand(rh, rw)
    i = torch.arange(rh, device="cuda", dtype=torch.float64)[:, None].expand(rh, rw)

    def position(th, cam, col, row):
        A = ir[cam]
        X = [A[r, 0] * col + A[r, 1] * row + A[r, 2] for r in range(3)]
        if cam == 1:
            # E^T X for E = exp([rot]x), at rot = 0 to first order (X + X x rot)
            e = th[13:16]
            X = [X[0] + X[1] * e[2] - X[2] * e[1], X[1] + X[2] * e[0] - X[0] * e[2], X[2] + X[0] * e[1] - X[1] * e[0]]
        x, y = X[0] / X[2], X[1] / X[2]
        c = th[6 * cam:6 * cam + 6]
        r2 = x * x + y * y
        s = 1 + r2 * (c[4] + r2 * c[5])
        return c[0] * x * s + c[2], c[1] * y * s + c[3]

    total = dict(loss=0.0, n_points=0.0, grad=torch.zeros(16, dtype=torch.float64, device="cuda"),
                 jtj=torch.zeros((16, 16), dtype=torch.float64, device="cuda"))
    th0 = torch.tensor(theta, device="cuda", dtype=torch.float64)
    for order, res, best, plane in views:
        ok = (best >= 1) & (best + 1 < rw)
        corner = []
        cols = [j, best - 1.0, best + 0.0, best + 1.0]
        for s, col in enumerate(cols):
            cam = 0 if s == 0 else 1
            u, v = position(th0, cam, col, i)
            ok &= (u >= 0) & (v >= 0) & (u < W - 1) & (v < H - 1)
            x0, y0 = u.clamp(0, W - 2).floor().to(torch.int64), v.clamp(0, H - 2).floor().to(torch.int64)
            k = [order[cam][y0 + b, x0 + a] for b in (0, 1) for a in (0, 1)]
            ph = [TWO_PI * kk.to(torch.float64) + res[cam][y0 + b, x0 + a].to(torch.float64)
                  for kk, (b, a) in zip(k, ((0, 0), (0, 1), (1, 0), (1, 1)))]
            for kk in k:
                ok &= kk >= 1
            corner.append((x0.to(torch.float64), y0.to(torch.float64), ph))

        def inverse_depth(th):
            smp = []
            for s, col in enumerate(cols):
                u, v = position(th, 0 if s == 0 else 1, col, i)
                x0, y0, ph = corner[s]
                a, b = u - x0, v - y0
                smp.append((1 - b) * ((1 - a) * ph[0] + a * ph[1]) + b * ((1 - a) * ph[2] + a * ph[3]))
            c0, c1, c2 = (p - smp[0] for p in smp[1:])
            den = 2 * (c0 - c1) * (c1 - c2)
            delta = torch.where(den.abs() > 1e-9, c1 * (c0 - c2) / torch.where(den.abs() > 1e-9, den, 1.0), 0.0)
            d = j - best - delta
            Tx = Tx0 * th[12] / B0
            return (dcx - d) / Tx, d

        w, d = inverse_depth(th0)
        z = Q[2, 3] / w
        ok &= (d.abs() >= 1e-5) & (z > zmin) & (z < zmax)
        nP = (plane[0] * (j + Q[0, 3]) + plane[1] * (i + Q[1, 3]) + plane[2] * Q[2, 3]) / w
        r = torch.where(ok, nP + plane[3], 0.0)
        total["loss"] += float((r * r).sum())
        total["n_points"] += float(ok.sum())
        J = torch.empty((16, rh * rw), dtype=torch.float64, device="cuda")
        for a in range(16):
            t = torch.zeros_like(th0)
            t[a] = 1.0
            _, (dw, _) = torch.func.jvp(inverse_depth, (th0,), (t,))
            J[a] = torch.where(ok, -nP / w * dw, 0.0).reshape(-1)
        total["grad"] += 2.0 * (J @ r.reshape(-1))
        total["jtj"] += J @ J.T
        del J
    return {"loss": total["loss"], "n_points": total["n_points"], "grad": total["grad"].cpu().numpy(),
            "jtj": total["jtj"].cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "pair":
        return None  # whole pipelines: the stages' cases hold their values
    if kind == "decode":
        spec = _spec(case["encoding"], case["width"], case["height"], seed + 1, case["hdr"])
        k, r, ok, mod = _decode64(_frames(spec, 0), spec, case["hdr"])
        return {"order": None, "residual": torch.where(ok, r, 0.0), "mod": None if case["hdr"] else mod, "valid": None}
    if kind in ("rectify_match", "reconstructor"):
        spec = _spec("hier", case["width"], case["height"], seed + 1)
        left, right = _decoded_pair(spec)
        ctx = _context(spec)
        disp = _match64(ctx, spec.rig, left, right, spec.pha_f)
        return disp if kind == "rectify_match" else (_reconstruct64(ctx, disp, radius=case["radius"]), None)
    if kind in ("sor", "mls", "metric_gaussian"):
        ctx = _cloud_context(case)
        xyz, mask = _cloud(ctx, seed)
        if kind == "sor":
            return None, _sor64(ctx, xyz, mask, case["mean_k"])
        if kind == "mls":
            return _mls64(ctx, xyz, mask, case)
        return _metric_gaussian64(ctx, xyz, mask, case["sigma"])
    spec, ctx, views, theta = _diff_inputs(case, seed)
    return _diff64(spec, ctx, views, theta)

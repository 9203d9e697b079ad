"""The post-smooth, the pixel Gaussian and the radius filter at sizes around their
strips (30 columns), row bands and tiles (32 x 32 and 32 x 8 pixels): the smooth
through the f64 phase map's own blur, the filters against their definitions in
64 bits.  A pair within float rounding of a threshold may fall either way."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (3, 29), (7, 30), (33, 31), (40, 61), (70, 97)]


def _cloud(rows, cols):
    g = np.random.default_rng(rows * 1000 + cols)
    u, v = np.meshgrid(np.arange(cols), np.arange(rows))
    xyz = np.stack([u + g.normal(0, 0.2, u.shape), v + g.normal(0, 0.2, u.shape), 900 + g.normal(0, 0.5, u.shape)], -1)
    mask = (g.random((rows, cols)) < 0.85).astype(np.uint8)
    xyz[mask == 0] = 0
    return xyz.astype(np.float32), mask


@pytest.mark.parametrize("rows,cols", SIZES)
@pytest.mark.parametrize("window,nb", [(1, 0), (4, 5), (10, 10), (31, 40), (96, 60)])
def test_ror_tiles(ctx, rows, cols, window, nb):
    from zim_gb300 import api
    xyz, mask = _cloud(rows, cols)
    r = np.float32(2.6 if nb < 40 else 5.3)
    out, mo = (t.cpu().numpy() for t in api.filter_ror(ctx, torch.from_numpy(xyz).cuda(), torch.from_numpy(mask).cuda(),
                                                       float(r), nb, window))
    hw = window // 2
    p = np.full((rows + 2 * hw, cols + 2 * hw, 3), np.nan)
    p[hw:hw + rows, hw:hw + cols] = np.where(mask[..., None] > 0, xyz, np.nan)
    cnt, near = np.zeros((rows, cols), int), np.zeros((rows, cols), bool)
    for i in range(2 * hw + 1):
        for j in range(2 * hw + 1):
            if i != hw or j != hw:
                d2 = ((p[i:i + rows, j:j + cols] - xyz) ** 2).sum(-1)
                cnt += d2 <= float(r) ** 2
                near |= np.abs(d2 - float(r) ** 2) < 1e-4
    keep = (mask > 0) & (cnt >= nb)
    assert np.array_equal((mo > 0)[~near], keep[~near])
    assert np.array_equal(out, np.where(mo[..., None] > 0, xyz, 0))


@pytest.mark.parametrize("rows,cols", SIZES)
def test_px_gaussian_strips(ctx, rows, cols):
    from zim_gb300 import api
    xyz, mask = _cloud(rows, cols)
    out, mo = (t.cpu().numpy() for t in api.filter_px_gaussian(ctx, torch.from_numpy(xyz).cuda(),
                                                               torch.from_numpy(mask).cuda(), True))
    e = np.exp(-0.5 / 0.49)
    k = np.array([e, 1, e]) / (1 + 2 * e)
    acc, cnt = np.zeros((rows, cols, 3)), np.zeros((rows, cols))
    p, m = np.pad(xyz.astype(np.float64), ((1, 1), (1, 1), (0, 0))), np.pad(mask, 1)
    near = np.zeros((rows, cols), bool)
    for i in range(3):
        for j in range(3):
            q = p[i:i + rows, j:j + cols]
            dx = np.abs(q[..., 0] - xyz[..., 0])
            w = np.where((m[i:i + rows, j:j + cols] > 0) & (dx < 3.0), k[i] * k[j], 0.0)
            near |= np.abs(dx - 3.0) < 1e-4
            acc += w[..., None] * q
            cnt += w
    inner = np.zeros((rows, cols), bool)
    inner[1:-1, 1:-1] = True
    near |= np.abs(cnt - 0.8) < 1e-5
    keep = (mask > 0) & inner & (cnt > 0.8)
    assert np.array_equal((mo > 0)[~near], keep[~near])
    sel = keep & ~near
    ref = acc[sel] / cnt[sel][:, None]
    # two float ulps of the largest coordinate, as for the filters' other parity tests
    assert (np.abs(out[sel] - ref) <= 1e-5 + 2 * np.spacing(np.float32(1000.0))).all()


@pytest.mark.parametrize("rows,cols", SIZES)
@pytest.mark.parametrize("hdr", [False, True])
def test_post_smooth_strips(native, rows, cols, hdr):
    """Identity rectification: the rectified phase is the post-smoothed one, which
    zim_decode_phase_f64 forms by itself in FP64."""
    from zim_gb300 import api, synth
    c = api.Context(0)
    c.set_calibration(synth.make_rig(cols, rows, 500.0, 50.0).as_dict(), False)
    g = np.random.default_rng(rows + 7 * cols)
    k = g.integers(0, 120, (rows, cols)).astype(np.int32)
    r = g.uniform(-3.1, 3.1, (rows, cols)).astype(np.float32)
    if hdr:
        bad = g.random((rows, cols)) < 0.3
        k[bad], r[bad] = -1, 0
    kt, rt = torch.from_numpy(k).cuda(), torch.from_numpy(r).cuda()
    ref = api.decode_phase_f64(c, kt, rt, True, hdr).cpu().numpy()
    mode = 2 if hdr else 1
    base = torch.empty((rows, cols), dtype=torch.int32, device="cuda")
    res = torch.empty((rows, cols), dtype=torch.float32, device="cuda")
    ro = torch.empty_like(base)
    mx, my = (t.cpu().numpy() for t in c.rectify_maps(0))
    if np.abs(mx - np.arange(cols)[None]).max() > 1e-3 or np.abs(my - np.arange(rows)[:, None]).max() > 1e-3:
        pytest.skip("the rig's map is not the identity")
    c.check(c._L.zim_rectify(c.h, 0, api._p(kt), api._p(rt), rows, cols, mode, api._p(base), api._p(res), api._p(ro),
                             api._stream()))
    got = 2 * np.pi * base.cpu().numpy().astype(np.float64) + res.cpu().numpy()
    # FP32 residual sums of nine taps below 4 pi: a few roundings of 2^-24 relative
    assert np.abs(got - ref).max() <= 1e-5

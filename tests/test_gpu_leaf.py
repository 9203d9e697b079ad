"""The bounding-box tree searches (SOR's deferred queries, the metric Gaussian's
uncertified ones) against brute force in 64 bits, at sizes around the tree's
leaf (8 pixels) and node (64 pixels) edges, on dense and sparse clouds, with and
without pixel rays.  Tolerances: mean distances 1e-5 relative (the fixed-point
roots hold 2^-22 of the largest), smoothed points 1e-5 mm plus two float ulps of
the largest coordinate, as for the filters' other parity tests."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 70), (7, 9), (8, 64), (65, 63), (129, 66), (30, 200)]


def _cloud(rows, cols, fill, seed):
    """Points on pixel rays (f = 1000 px) of a rough surface; a few far off theirs."""
    g = np.random.default_rng(seed)
    z = 900.0 + g.normal(0, 0.5, (rows, cols)) + np.where(g.random((rows, cols)) < 0.02, -80.0, 0.0)
    u, v = np.meshgrid(np.arange(cols) - (cols - 1) / 2, np.arange(rows) - (rows - 1) / 2)
    xyz = np.stack([u * z / 1000.0, v * z / 1000.0, z], -1).astype(np.float32)
    far = g.random((rows, cols)) < 0.01
    xyz[far] += g.uniform(-60, 60, (int(far.sum()), 3)).astype(np.float32)
    mask = (g.random((rows, cols)) < fill).astype(np.uint8)
    xyz[mask == 0] = 0
    return xyz, mask


def _context(rows, cols, rays):
    from zim_gb300 import api, synth
    c = api.Context(0)
    if rays:
        c.set_calibration(synth.make_rig(cols, rows, 1000.0, 100.0).as_dict(), False)
        assert (c.rect_h, c.rect_w) == (rows, cols)
    return c


@pytest.mark.parametrize("rays", [False, True])
@pytest.mark.parametrize("fill", [0.08, 0.95])
@pytest.mark.parametrize("rows,cols", SIZES)
def test_tree_searches_match_brute_force(native, rows, cols, fill, rays):
    from zim_gb300 import api
    xyz, mask = _cloud(rows, cols, fill, 1000 * rows + cols)
    n = int(mask.sum())
    ctx = _context(rows, cols, rays)
    xt, mt = torch.from_numpy(xyz).cuda(), torch.from_numpy(mask).cuda()
    p = xyz[mask > 0].astype(np.float64)
    d = np.sqrt(((p[:, None] - p[None]) ** 2).sum(-1))
    for k in (1, 6, 63):
        if n <= k:
            continue
        _, md = api.filter_sor(ctx, xt, mt, k, 1.0, want_mean_dist=True)
        ref = np.sort(d, axis=1)[:, :k + 1].sum(1) / k
        got = md.cpu().numpy()[mask > 0]
        assert np.abs(got - ref).max() <= 1e-5 * ref.max()
        assert (np.abs(got - ref) <= 1e-5 * ref).all()
    sigma = 1.0
    w = np.where(d <= 3 * sigma, np.exp(-d * d / (2 * sigma * sigma)), 0.0)
    # a pair within float rounding of the cut-off may fall either way
    sure = (np.abs(d - 3 * sigma) > 1e-4).all(axis=1)
    ref = (w @ p) / w.sum(1, keepdims=True)
    got = api.filter_metric_gaussian(ctx, xt, mt, sigma).cpu().numpy()[mask > 0]
    tol = 1e-5 + 2 * np.spacing(np.abs(ref).max(axis=1, keepdims=True).astype(np.float32))
    assert (np.abs(got - ref) <= tol)[sure].all()
    assert ctx.check_device() == 0


@pytest.mark.parametrize("rows,cols", SIZES[1:])
@pytest.mark.parametrize("window,sigma,order,radius", [(1, 1.0, 1, 0.0), (5, 1.0, 2, 0.0), (13, 2.0, 0, 0.0),
                                                       (30, 1.2, 1, 0.0), (30, 6.0, 2, 16.0), (40, 1.5, 2, 4.0)])
def test_mls_ray_window_equals_full_window(native, rows, cols, window, sigma, order, radius):
    """The ray bound only leaves out pixels beyond the cut-off, staged in shared
    memory or read from global memory: the same bits as the full window (the
    cloud padded by an invalid column has no pixel rays)."""
    from zim_gb300 import api
    xyz, mask = _cloud(rows, cols, 0.95, 77 * rows + cols)
    xp = np.zeros((rows, cols + 1, 3), np.float32)
    mp = np.zeros((rows, cols + 1), np.uint8)
    xp[:, :cols], mp[:, :cols] = xyz, mask
    args = (window, sigma, order, radius, 2)
    a = api.filter_mls(_context(rows, cols, True), torch.from_numpy(xyz).cuda(), torch.from_numpy(mask).cuda(), *args)
    b = api.filter_mls(_context(rows, cols, False), torch.from_numpy(xp).cuda(), torch.from_numpy(mp).cuda(), *args)
    assert torch.equal(a, b[:, :cols].contiguous())
    assert not torch.equal(a.cpu(), torch.from_numpy(xyz))

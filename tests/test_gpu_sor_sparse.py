"""SOR on sparse clouds, whose windows hold fewer than k + 1 points: the tree search is
bounded by the leaves around the query (up to 3, then 7 on either side) or, with too few
points there, by the nodes.  Mean distances against brute force in 64 bits, 1e-5
relative (the fixed-point roots hold 2^-22 of the largest); and a cloud with a tenth of
the points stays within a few times the full one's cost."""
import numpy as np
import pytest
import torch

from test_gpu_match_windows import _microseconds

pytestmark = pytest.mark.gpu


def _cloud(rows, cols, fill, seed):
    g = np.random.default_rng(seed)
    z = 900.0 + g.normal(0, 0.3, (rows, cols)) + np.where(np.arange(cols) > cols // 2, 20.0, 0.0)
    u, v = np.meshgrid(np.arange(cols) - (cols - 1) / 2, np.arange(rows) - (rows - 1) / 2)
    xyz = np.stack([u * z / 1000.0, v * z / 1000.0, z], -1).astype(np.float32)
    return xyz, (g.random((rows, cols)) < fill).astype(np.uint8)


def _context(rows, cols, rays):
    from zim_gb300 import api, synth
    ctx = api.Context(0)
    if rays:
        ctx.set_calibration(synth.make_rig(cols, rows, 1000.0, 100.0).as_dict(), False)
        assert (ctx.rect_h, ctx.rect_w) == (rows, cols)
    return ctx


@pytest.mark.parametrize("rays", [False, True])
@pytest.mark.parametrize("fill", [0.003, 0.01, 0.03, 0.1])
@pytest.mark.parametrize("rows,cols", [(56, 57), (121, 130), (230, 300)])
def test_sparse_against_brute_force(native, rows, cols, fill, rays):
    from zim_gb300 import api
    xyz, mask = _cloud(rows, cols, fill, rows)
    mask[0, 0] = mask[-1, -1] = mask[rows // 2, cols // 2] = 1
    ctx = _context(rows, cols, rays)
    p = torch.from_numpy(xyz[mask > 0]).cuda().double()
    d = torch.cdist(p, p, compute_mode="donot_use_mm_for_euclid_dist").sort(dim=1).values
    for k in (2, 9, 40, 63):
        if len(p) <= k:
            continue
        _, md = api.filter_sor(ctx, torch.from_numpy(xyz).cuda(), torch.from_numpy(mask).cuda(), k, 1.0, want_mean_dist=True)
        ref = d[:, :k + 1].sum(1) / k
        got = md[torch.from_numpy(mask).cuda() > 0].double()
        assert ((got - ref).abs() <= 1e-5 * ref).all()
    assert ctx.check_device() == 0


def test_sparse_cost(native):
    """A tenth of a surface's points at 1626 x 1236 (0.375 mm a pixel) against six tenths."""
    from zim_gb300 import api, synth
    rows, cols = 1236, 1626
    ctx = api.Context(0)
    ctx.set_calibration(synth.make_rig(cols, rows, 2400.0, 100.0).as_dict(), False)
    g = np.random.default_rng(1)
    z = (900.0 + g.normal(0, 0.05, (rows, cols)) + 30.0 * np.sin(np.arange(cols) / 97.0)
         + np.where((np.arange(cols) // 200) % 2, 25.0, 0.0))
    u, v = np.meshgrid(np.arange(cols) - (cols - 1) / 2, np.arange(rows) - (rows - 1) / 2)
    xyz = torch.from_numpy(np.stack([u * z / 2400.0, v * z / 2400.0, z], -1).astype(np.float32)).cuda()
    r = g.random((rows, cols))
    t = []
    for fill in (0.1, 0.6):
        mask = torch.from_numpy((r < fill).astype(np.uint8)).cuda()
        t.append(_microseconds(lambda: api.filter_sor(ctx, xyz, mask, 30, 1.0)))
    assert t[0] <= 5.5 * t[1], t

"""The window pass of the statistical outlier filter keeps the k + 1 nearest in
groups of five: k at a group's edges, over a cloud whose window holds invalid
pixels, off-ray points, equal distances and fewer than k + 1 points, against brute
force in 64 bits and, bit for bit, against the search without pixel rays (both sum
the same k + 1 roots in fixed point).  1e-5 relative as for the filter's other
parity tests (the fixed-point roots hold 2^-22 of the largest)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS, COLS = 37, 50  # no multiple of the 16 x 16 tiles


def _cloud():
    g = np.random.default_rng(5)
    z = 900.0 + g.normal(0, 0.3, (ROWS, COLS)) + np.where(np.arange(COLS) > 30, 4.0, 0.0)
    u, v = np.meshgrid(np.arange(COLS) - (COLS - 1) / 2, np.arange(ROWS) - (ROWS - 1) / 2)
    xyz = np.stack([u * z / 1000.0, v * z / 1000.0, z], -1).astype(np.float32)
    xyz[20:27, 5:12] = xyz[23, 8]  # equal points: equal distances
    xyz[5, 40:44] += 25.0          # off their rays
    mask = (g.random((ROWS, COLS)) < 0.9).astype(np.uint8)
    mask[0:14, 0:14] = 0
    mask[4, 4:7] = 1               # fewer than k + 1 points in the window
    xyz[mask == 0] = 0
    return xyz, mask


@pytest.mark.parametrize("k", [1, 3, 4, 5, 8, 9, 10, 14, 29, 30, 49, 50, 59, 60, 63])
def test_near_set(native, k):
    from zim_gb300 import api, synth
    xyz, mask = _cloud()
    xt, mt = torch.from_numpy(xyz).cuda(), torch.from_numpy(mask).cuda()
    ray, plain = api.Context(0), api.Context(0)
    ray.set_calibration(synth.make_rig(COLS, ROWS, 1000.0, 100.0).as_dict(), False)
    assert (ray.rect_h, ray.rect_w) == (ROWS, COLS)
    mo, md = api.filter_sor(ray, xt, mt, k, 1.0, want_mean_dist=True)
    mo2, md2 = api.filter_sor(plain, xt, mt, k, 1.0, want_mean_dist=True)
    assert torch.equal(md, md2) and torch.equal(mo, mo2)
    p = xyz[mask > 0].astype(np.float64)
    d = np.sqrt(((p[:, None] - p[None]) ** 2).sum(-1))
    ref = np.sort(d, axis=1)[:, :k + 1].sum(1) / k
    assert (np.abs(md.cpu().numpy()[mask > 0] - ref) <= 1e-5 * ref).all()

"""MLS with pixel rays on small clouds, at half-windows on both sides of the rules that
stage the window whole (12; 24 with one wave of tiles; 30 with a few tiles), with points
off their rays: the bits of the search without rays.  Just beyond 12 the cost of a small
cloud stays near that at 12."""
import numpy as np
import pytest
import torch

from test_gpu_match_windows import _microseconds

pytestmark = pytest.mark.gpu


def _cloud(rows, cols, off):
    g = np.random.default_rng(rows)
    z = 900.0 + g.normal(0, 0.2, (rows, cols)) + np.where(np.arange(cols) > 2 * cols // 3, 3.0, 0.0)
    u, v = np.meshgrid(np.arange(cols) - (cols - 1) / 2, np.arange(rows) - (rows - 1) / 2)
    xyz = np.stack([u * z / 1000.0, v * z / 1000.0, z], -1).astype(np.float32)
    mask = (g.random((rows, cols)) < 0.93).astype(np.uint8)
    if off:
        xyz[rows // 2, cols // 2, 0] += 25.0
        xyz[0, 0] = np.nan
        mask[[rows // 2, 0], [cols // 2, 0]] = 1
    return torch.from_numpy(xyz).cuda(), torch.from_numpy(mask).cuda()


def _contexts(rows, cols):
    from zim_gb300 import api, synth
    ray = api.Context(0)
    ray.set_calibration(synth.make_rig(cols, rows, 1000.0, 100.0).as_dict(), False)
    assert (ray.rect_h, ray.rect_w) == (rows, cols)
    return ray, api.Context(0)


@pytest.mark.parametrize("rows,cols", [(1, 17), (33, 47), (64, 79), (330, 400)])
@pytest.mark.parametrize("window", [12, 13, 20, 24, 25, 30, 31])
@pytest.mark.parametrize("off", [False, True])
def test_staged_whole(native, rows, cols, window, off):
    from zim_gb300 import api
    xyz, mask = _cloud(rows, cols, off)
    ray, plain = _contexts(rows, cols)
    for order in (1, 2):
        a = api.filter_mls(ray, xyz, mask, window, 0.9, order, 2.5, 1)
        b = api.filter_mls(plain, xyz, mask, window, 0.9, order, 2.5, 1)
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
        assert rows == 1 or not torch.equal(a, xyz)


def test_small_cloud_beyond_twelve(native):
    from zim_gb300 import api
    xyz, mask = _cloud(64, 64, False)
    ray, _ = _contexts(64, 64)
    t = [_microseconds(lambda: api.filter_mls(ray, xyz, mask, w, 0.6, 1, 1.8, 1)) for w in (12, 13)]
    assert t[1] <= 1.3 * t[0], t

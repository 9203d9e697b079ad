"""MLS with pixel rays at half-windows around the rules that choose its kernel (7:
the whole window; 12: tiles that need more are done apart, a few rows at a time),
on a cloud where some tiles need a few pixels and others, with points far off
their rays or without finite coordinates, all of the window.  The neighbours and
their order are those of the full window, so the bits are those of the search
without rays."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS, COLS = 53, 90


def _cloud():
    g = np.random.default_rng(9)
    z = 900.0 + g.normal(0, 0.2, (ROWS, COLS)) + np.where(np.arange(COLS) > 60, 3.0, 0.0)
    u, v = np.meshgrid(np.arange(COLS) - (COLS - 1) / 2, np.arange(ROWS) - (ROWS - 1) / 2)
    xyz = np.stack([u * z / 1000.0, v * z / 1000.0, z], -1).astype(np.float32)
    mask = (g.random((ROWS, COLS)) < 0.93).astype(np.uint8)
    xyz[3, 2:5, 0] += 30.0
    xyz[50, 4] = np.nan
    xyz[51, 88, 1] = np.inf
    mask[[3, 3, 3, 50, 51], [2, 3, 4, 4, 88]] = 1
    return torch.from_numpy(xyz).cuda(), torch.from_numpy(mask).cuda()


@pytest.mark.parametrize("window", [7, 8, 12, 13, 30, 64])
@pytest.mark.parametrize("order,radius,iterations", [(0, 2.5, 1), (1, 2.5, 2), (2, 2.5, 1), (2, 14.0, 1)])
def test_windows(native, window, order, radius, iterations):
    from zim_gb300 import api, synth
    xyz, mask = _cloud()
    ray, plain = api.Context(0), api.Context(0)
    ray.set_calibration(synth.make_rig(COLS, ROWS, 1000.0, 100.0).as_dict(), False)
    assert (ray.rect_h, ray.rect_w) == (ROWS, COLS)
    a = api.filter_mls(ray, xyz, mask, window, 1.5, order, radius, iterations)
    b = api.filter_mls(plain, xyz, mask, window, 1.5, order, radius, iterations)
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert not torch.equal(a, xyz)

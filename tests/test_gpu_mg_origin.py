"""The metric Gaussian on what the pixel Gaussian leaves: valid points at the origin
along the image's border, all each other's neighbours.  They stay where they are, the
surface comes out as without them, and they cost no more than a few times a dense
surface that is searched as a whole."""
import numpy as np
import pytest
import torch

from test_gpu_match_windows import _microseconds

pytestmark = pytest.mark.gpu


def _cloud(rows, cols):
    g = np.random.default_rng(rows)
    z = (900.0 + g.normal(0, 0.05, (rows, cols)) + 30.0 * np.sin(np.arange(cols) / 97.0)
         + np.where((np.arange(cols) // 200) % 2, 25.0, 0.0))
    u, v = np.meshgrid(np.arange(cols) - (cols - 1) / 2, np.arange(rows) - (rows - 1) / 2)
    xyz = torch.from_numpy(np.stack([u * z / 2400.0, v * z / 2400.0, z], -1).astype(np.float32)).cuda()
    border = torch.ones((rows, cols), dtype=torch.bool, device="cuda")
    border[1:-1, 1:-1] = False
    return xyz, border


def _contexts(rows, cols):
    from zim_gb300 import api, synth
    ray = api.Context(0)
    ray.set_calibration(synth.make_rig(cols, rows, 2400.0, 100.0).as_dict(), False)
    assert (ray.rect_h, ray.rect_w) == (rows, cols)
    return ray, api.Context(0)


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 40), (17, 33), (70, 129), (200, 300)])
def test_border_at_the_origin(native, rows, cols):
    from zim_gb300 import api
    xyz, border = _cloud(rows, cols)
    xyz[border] = 0
    mask = torch.ones((rows, cols), dtype=torch.uint8, device="cuda")
    inside = torch.where(border, 0, 1).to(torch.uint8)
    for ctx in _contexts(rows, cols):
        out, ref = api.filter_metric_gaussian(ctx, xyz, mask, 0.5), api.filter_metric_gaussian(ctx, xyz, inside, 0.5)
        assert bool((out[border] == 0).all())
        if bool(inside.any()):
            # a window sum and the tree's 64-bit sum of the same points: 1e-5 mm and two float steps
            tol = 1e-5 + 2 * np.spacing(np.float32(xyz.abs().max().item()))
            assert (out[inside > 0] - ref[inside > 0]).abs().max() <= tol


def test_border_cost(native):
    from zim_gb300 import api
    rows, cols = 768, 1024
    ray, plain = _contexts(rows, cols)
    xyz, border = _cloud(rows, cols)
    dense = (torch.rand((rows, cols), device="cuda") < 0.6).to(torch.uint8)
    surface = _microseconds(lambda: api.filter_metric_gaussian(plain, xyz, dense, 0.5))
    xyz[border] = 0
    ring = border.to(torch.uint8)
    assert _microseconds(lambda: api.filter_metric_gaussian(ray, xyz, ring, 0.5)) <= 8 * surface

"""The metric Gaussian on a cloud with valid points whose coordinates are not all
finite: they stay as they are, and the others come out as if those were invalid."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rays", [False, True])
@pytest.mark.parametrize("rows,cols", [(9, 17), (40, 70)])
def test_points_without_finite_coordinates(native, rows, cols, rays):
    from zim_gb300 import api, synth
    g = np.random.default_rng(rows)
    z = 900.0 + g.normal(0, 0.3, (rows, cols))
    u, v = np.meshgrid(np.arange(cols) - (cols - 1) / 2, np.arange(rows) - (rows - 1) / 2)
    xyz = torch.from_numpy(np.stack([u * z / 1000.0, v * z / 1000.0, z], -1).astype(np.float32)).cuda()
    mask = torch.ones((rows, cols), dtype=torch.uint8, device="cuda")
    ctx = api.Context(0)
    if rays:
        ctx.set_calibration(synth.make_rig(cols, rows, 1000.0, 100.0).as_dict(), False)
        assert (ctx.rect_h, ctx.rect_w) == (rows, cols)
    bad = [(0, 0), (rows // 2, cols // 2), (rows - 1, 3)]
    for k, (p, q) in enumerate(bad):
        xyz[p, q, k] = (float("nan"), float("inf"), -float("inf"))[k]
    out = api.filter_metric_gaussian(ctx, xyz, mask, 0.8)
    without = mask.clone()
    for p, q in bad:
        assert torch.equal(out[p, q].view(torch.int32), xyz[p, q].view(torch.int32))
        without[p, q] = 0
    ref = api.filter_metric_gaussian(ctx, xyz, without, 0.8)
    keep = without > 0
    assert torch.isfinite(out[keep]).all()
    assert (out[keep] - ref[keep]).abs().max() <= 1e-3  # one float ulp of 900 mm is 6e-5 mm

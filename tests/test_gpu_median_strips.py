"""The 5x5 median + reprojection at widths around its 58-column strips and heights
around its row bands: the median is exact selection with replicated borders, so it
equals numpy's to the bit, and the points match the FP64 formula within a few FP32
roundings."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 1), (2, 3), (5, 57), (9, 58), (33, 59), (70, 116), (6, 117), (40, 175)])
@pytest.mark.parametrize("median", [0, 1])
def test_median_strip_edges(native, rows, cols, median):
    from zim_gb300 import api, synth
    ctx = api.Context(0)
    ctx.set_calibration(synth.make_rig(640, 480, 1000.0, 100.0).as_dict(), False)
    g = np.random.default_rng(rows * 1000 + cols)
    d = (1000.0 * 100.0 / g.uniform(700, 1100, (rows, cols))).astype(np.float32)
    d[g.random((rows, cols)) < 0.3] = 0
    d[g.random((rows, cols)) < 0.2] = np.float32(123.5)  # ties
    cfg = api.recon_config(use_disp_median_filter=median, max_depth=1000.0)
    dm, xyz, mask = (t.cpu().numpy() for t in api.median_reproject(ctx, cfg, torch.from_numpy(d).cuda()))
    if median:
        p = np.pad(d, 2, mode="edge")
        ref = np.median(np.stack([p[i:i + rows, j:j + cols] for i in range(5) for j in range(5)]), axis=0)
    else:
        ref = d
    assert np.array_equal(dm, ref.astype(np.float32))
    w = np.float64(ctx.Q[3, 2]) * dm.astype(np.float64) + ctx.Q[3, 3]
    w[w == 0] = 1e-30
    z = ctx.Q[2, 3] / w
    x = (np.arange(cols)[None] + ctx.Q[0, 3]) / w
    sure = np.abs(z - 1000.0) > 1e-3
    ok = (np.abs(dm) >= 1e-5) & (z > 0) & (z < 1000.0)
    assert np.array_equal((mask > 0)[sure], ok[sure])
    both = ok & (mask > 0)
    # FP32 reprojection: a few roundings of 2^-24 relative
    assert (np.abs(xyz[..., 2] - z) <= 1e-6 * z)[both].all()
    assert (np.abs(xyz[..., 0] - x) <= 1e-6 * np.abs(x) + 1e-6 * 1000)[both].all()
    assert (xyz[mask == 0] == 0).all()

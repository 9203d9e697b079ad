"""SOR on clouds with valid points whose coordinates are not all finite (nobody's
neighbours: the others' mean distances are those without them, their own is 0 and the
error word says so), with and without pixel rays, the metric Gaussian beside it; and
SOR on buffers that do not lie on whole vector loads, whose statistics are the same
bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cloud(rows, cols):
    g = np.random.default_rng(rows)
    z = 900.0 + g.normal(0, 0.3, (rows, cols))
    u, v = np.meshgrid(np.arange(cols) - (cols - 1) / 2, np.arange(rows) - (rows - 1) / 2)
    xyz = torch.from_numpy(np.stack([u * z / 1000.0, v * z / 1000.0, z], -1).astype(np.float32)).cuda()
    return xyz, torch.from_numpy((g.random((rows, cols)) < 0.96).astype(np.uint8)).cuda()


def _context(rows, cols, rays):
    from zim_gb300 import api, synth
    ctx = api.Context(0)
    if rays:
        ctx.set_calibration(synth.make_rig(cols, rows, 1000.0, 100.0).as_dict(), False)
        assert (ctx.rect_h, ctx.rect_w) == (rows, cols)
    return ctx


@pytest.mark.parametrize("rays", [False, True])
@pytest.mark.parametrize("bad", ["nan", "inf", "mixed"])
@pytest.mark.parametrize("rows,cols", [(20, 37), (48, 90)])
def test_points_without_finite_coordinates(native, rows, cols, bad, rays):
    from zim_gb300 import _lib, api
    xyz, mask = _cloud(rows, cols)
    at = torch.zeros((rows, cols), dtype=torch.bool, device="cuda")
    at[rows // 2, 2:-2] = True  # more of them than neighbours asked for
    at[0, 0] = at[-1, -1] = True
    mask[at] = 1
    nan, inf = float("nan"), float("inf")
    values = {"nan": [[nan] * 3], "inf": [[inf] * 3], "mixed": [[nan, 0.0, 900.0], [0.0, -inf, 900.0], [inf, nan, -inf]]}[bad]
    fill = torch.tensor([values[i % len(values)] for i in range(int(at.sum()))], device="cuda")
    xyz[at] = fill
    without = mask.clone()
    without[at] = 0
    keep = without > 0
    for k in (6, 20):
        ctx = _context(rows, cols, rays)
        _, md = api.filter_sor(ctx, xyz, mask, k, 1.0, want_mean_dist=True)
        stats = api.sor_stats(ctx)
        _, ref = api.filter_sor(_context(rows, cols, rays), xyz, without, k, 1.0, want_mean_dist=True)
        assert torch.equal(md[keep], ref[keep]) and bool((ref[keep] > 0).all())
        assert bool((md[at] == 0).all())
        assert np.isfinite(stats["threshold"]) and stats["n_valid"] == int(mask.sum())
        with pytest.raises(_lib.ZimError, match="0x00000010"):
            ctx.check_device()
    ctx = _context(rows, cols, rays)
    out, ref = api.filter_metric_gaussian(ctx, xyz, mask, 0.8), api.filter_metric_gaussian(ctx, xyz, without, 0.8)
    assert torch.equal(out[at].view(torch.int32), xyz[at].view(torch.int32))
    # a window sum and the tree's 64-bit sum of the same points: 1e-5 mm and two float steps
    tol = 1e-5 + 2 * np.spacing(np.float32(xyz[keep].abs().max().item()))
    assert (out[keep] - ref[keep]).abs().max() <= tol
    assert ctx.check_device() == 0


@pytest.mark.parametrize("rows,cols", [(37, 53), (300, 401)])
def test_statistics_do_not_depend_on_the_buffers_address(native, rows, cols):
    from zim_gb300 import api
    ctx = _context(rows, cols, True)
    xyz, mask = _cloud(rows, cols)
    # mean distances from a fraction of a millimetre to kilometres: their sums round
    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    far = torch.rand((rows, cols), generator=g, device="cuda") < 0.02
    xyz[..., 2] += torch.where(far, 1e7 * torch.rand((rows, cols), generator=g, device="cuda"), 0.0)
    odd = torch.empty(mask.numel() + 1, dtype=torch.uint8, device="cuda")[1:].view(mask.shape)
    odd.copy_(mask)
    a = api.filter_sor(ctx, xyz, mask, 20, 1.0, want_mean_dist=True)
    sa = api.sor_stats(ctx)
    b = api.filter_sor(ctx, xyz, odd, 20, 1.0, want_mean_dist=True)
    sb = api.sor_stats(ctx)
    assert sa == sb
    assert all(torch.equal(u, v) for u, v in zip(a, b))

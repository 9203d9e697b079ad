"""SOR on buffers that do not lie on whole vector loads: the statistics are the same
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

"""The adjoint with and without an upstream gradient (two kernels) and its view
loop at image sizes around the warp stride: a zero upstream gradient against none,
and several views in one call against the views one by one.  A gradient component
may differ by 1e-6 of sum |2 r J| <= 2 sqrt(loss * jtj_kk), a J^T J entry by 1e-6 of
the geometric mean of its diagonal entries: FP32 partial sums of a few dozen terms,
grouped differently."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _view(ctx, rows, cols, seed):
    from zim_gb300 import diff
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rh, rw = ctx.rect_h, ctx.rect_w
    orders, residuals = [], []
    for cam in (0, 1):
        x = torch.arange(cols, device="cuda", dtype=torch.float64)[None, :] + (8.0 if cam else 0.0)
        ph = 0.16 * (x + 40) + 0.01 * torch.randn((rows, cols), generator=g, device="cuda", dtype=torch.float64)
        k = torch.floor(ph / (2 * np.pi) + 0.5)
        ok = torch.rand((rows, cols), generator=g, device="cuda") < 0.98
        orders.append(torch.where(ok, k, 0.0).to(torch.int32))
        residuals.append((ph - 2 * np.pi * k).to(torch.float32))
    best = (torch.arange(rw, device="cuda")[None, :] - 8).expand(rh, rw).to(torch.int32).contiguous()
    return diff.View(orders, residuals, best, (0.02, -0.01, 0.99, -900.0 - seed))


@pytest.mark.parametrize("rows,cols", [(3, 40), (17, 33), (31, 100), (64, 257)])
def test_gradient_paths_and_views(native, rows, cols):
    from zim_gb300 import api, diff, synth
    ctx = api.Context(0)
    ctx.set_calibration(synth.make_rig(cols, rows, 400.0, 18.0, dist=(-0.05, 0.01, 0, 0, 0)).as_dict(), True)
    theta = diff.nominal(ctx)
    views = [_view(ctx, rows, cols, s) for s in range(3)]
    args = (1.5, 1.0, 5000.0)
    one = [diff.backward(ctx, theta, [v], *args) for v in views]
    assert sum(o["n_points"] for o in one) > 0.3 * 3 * rows * max(1, cols - 12)
    allv = diff.backward(ctx, theta, views, *args)
    for v in views:
        v.grad_xyz = torch.zeros((ctx.rect_h, ctx.rect_w, 3), device="cuda")
    up = diff.backward(ctx, theta, views, *args)
    fwd = diff.forward(ctx, theta, views, *args[1:])
    for key in ("loss", "n_points"):
        total = sum(o[key] for o in one)
        assert abs(allv[key] - total) <= 1e-12 * abs(total)
        assert abs(up[key] - total) <= 1e-12 * abs(total) and abs(fwd[key] - total) <= 1e-12 * abs(total)
    scale = 1.5 * 2 * np.sqrt(allv["loss"] * np.diag(allv["jtj"])) + 1e-300
    assert (np.abs(allv["grad"] - sum(o["grad"] for o in one)) <= 1e-6 * scale).all()
    assert (np.abs(allv["grad"] - up["grad"]) <= 1e-6 * scale).all()
    d = np.sqrt(np.outer(np.diag(allv["jtj"]), np.diag(allv["jtj"]))) + 1e-300
    assert (np.abs(allv["jtj"] - sum(o["jtj"] for o in one)) <= 1e-6 * d).all()
    assert (np.abs(allv["jtj"] - up["jtj"]) <= 1e-6 * d).all()
    assert np.array_equal(allv["jtj"], allv["jtj"].T)

"""The adjoint's sums over many views: 4096 times one view against 4096 times its sums.
All terms of a component have one sign here, so the sum of their magnitudes is at most
2 w sqrt(loss jtj_kk) (gradient) or sqrt(jtj_aa jtj_bb) (J^T J), and FP64 sums of a
lane's 16 x 4096 terms are within 65536 x 2^-53 of it."""
import numpy as np
import pytest
import torch

from test_gpu_diff_blocks import _view

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("upstream", [False, True])
@pytest.mark.parametrize("rows,cols", [(64, 64), (48, 50)])
def test_many_views(native, rows, cols, upstream):
    from zim_gb300 import api, diff, synth
    ctx = api.Context(0)
    ctx.set_calibration(synth.make_rig(cols, rows, 400.0, 18.0).as_dict(), False)
    assert (ctx.rect_h, ctx.rect_w) == (rows, cols) and rows * cols % 32 == 0  # the same sets of 32 in every view
    view = _view(ctx, rows, cols, 3)
    view.plane = (0.02, -0.01, 0.99, -600.0)
    if upstream:
        view.grad_xyz = torch.zeros((rows, cols, 3), device="cuda")
    theta = diff.nominal(ctx)
    args = (1.5, 1.0, 5000.0)
    n = 4096
    one, many = diff.backward(ctx, theta, [view], *args), diff.backward(ctx, theta, [view] * n, *args)
    assert one["n_points"] > 0.5 * rows * cols and many["n_points"] == n * one["n_points"]
    tol = 65536 * 2.0 ** -53
    assert abs(many["loss"] - n * one["loss"]) <= tol * n * one["loss"]
    d = np.sqrt(np.diag(one["jtj"]))
    assert (np.abs(many["grad"] - n * one["grad"]) <= tol * n * 2 * 1.5 * np.sqrt(one["loss"]) * d).all()
    assert (np.abs(many["jtj"] - n * one["jtj"]) <= tol * n * np.outer(d, d)).all()

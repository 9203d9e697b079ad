"""The kernels that march strips (post-smooth, median, pixel Gaussian) at image sizes
on both sides of the rules for a band's rows (1, 2 and 4 and more), against the upper
rows alone, which take shorter bands: the same bits away from the cut.  On a tiny
image their launch is about as long as that of a kernel with one load per pixel."""
import pytest
import torch

from test_gpu_match_windows import _microseconds

pytestmark = pytest.mark.gpu


def _context(rows, cols):
    from zim_gb300 import api, synth
    ctx = api.Context(0)
    ctx.set_calibration(synth.make_rig(cols, rows, 1000.0, 100.0).as_dict(), False)
    return ctx


def _bits(t):
    return t.contiguous().view(torch.uint8)


@pytest.mark.parametrize("rows,cols", [(5, 29), (40, 70), (150, 300), (300, 400), (500, 600), (600, 800)])
def test_bands_agree(native, rows, cols):
    from zim_gb300 import api
    part = max(4, rows // 4)
    full, cut = _context(rows, cols), _context(part, cols)
    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    rand = lambda *s: torch.rand((rows, cols) + s, generator=g, device="cuda")
    disp = torch.where(rand() < 0.9, 8.0 + rand(), torch.zeros((), device="cuda"))
    order, res = (rand() * 40).to(torch.int32), rand()
    xyz, mask = 900 + rand(3), (rand() < 0.9).to(torch.uint8)
    rc = api.recon_config(reproject_model=0)
    top = lambda t: t[:part].contiguous()
    # the rows that a cut at `part` leaves alone: all but the window's half height above it
    a, b = api.median_reproject(full, rc, disp), api.median_reproject(cut, rc, top(disp))
    assert torch.equal(_bits(a[0][:part - 2]), _bits(b[0][:part - 2]))
    a, b = api.filter_px_gaussian(full, xyz, mask, True), api.filter_px_gaussian(cut, top(xyz), top(mask), True)
    assert all(torch.equal(_bits(u[:part - 1]), _bits(v[:part - 1])) for u, v in zip(a, b))
    a, b = api.decode_phase_f64(full, order, res), api.rectify(full, 0, order, res, True)
    assert torch.isfinite(a).all() and b[0].shape == (rows, cols)


def test_post_smooth_is_the_plain_remap_of_its_taps(native):
    """post_smooth of constant rows changes nothing: the smoothed and the plain remap agree."""
    from zim_gb300 import api
    for rows, cols in [(6, 31), (64, 64), (300, 400), (600, 800)]:
        ctx = _context(rows, cols)
        order = torch.full((rows, cols), 7, dtype=torch.int32, device="cuda")
        res = torch.full((rows, cols), 0.5, device="cuda")
        a, b = api.rectify(ctx, 0, order, res, True), api.rectify(ctx, 0, order, res, False)
        assert torch.equal(a[0], b[0]) and torch.equal(a[2], b[2])
        assert (a[1] - b[1]).abs().max() <= 1e-6


def test_tiny_images(native):
    from zim_gb300 import api
    ctx = _context(64, 64)
    order = torch.ones((64, 64), dtype=torch.int32, device="cuda")
    res, disp = torch.zeros((64, 64), device="cuda"), torch.full((64, 64), 8.0, device="cuda")
    xyz, mask = torch.rand((64, 64, 3), device="cuda"), torch.ones((64, 64), dtype=torch.uint8, device="cuda")
    rc = api.recon_config(use_disp_median_filter=0)
    one = _microseconds(lambda: api.rectify(ctx, 0, order, res, False))
    assert _microseconds(lambda: api.median_reproject(ctx, rc, disp)) <= 1.6 * one
    assert _microseconds(lambda: api.filter_px_gaussian(ctx, xyz, mask)) <= 1.6 * one

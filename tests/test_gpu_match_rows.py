"""The fused rectification and match against the two apart, bit for bit, at row
counts on both sides of the rule that chooses its block size (all rows in one wave
of the larger blocks) and at widths around the blocks' thread counts."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _side(rows, cols, shift, gen):
    x = torch.arange(cols, device="cuda", dtype=torch.float64)[None, :] + shift
    ph = 0.16 * (x + 40) + 0.02 * torch.randn((rows, cols), generator=gen, device="cuda", dtype=torch.float64)
    k = torch.floor(ph / 6.283185307179586 + 0.5)
    ok = torch.rand((rows, cols), generator=gen, device="cuda") < 0.98
    return torch.where(ok, k, 0.0).to(torch.int32), (ph - 6.283185307179586 * k).to(torch.float32)


@pytest.mark.parametrize("cols", [37, 257, 384, 385, 513])
@pytest.mark.parametrize("rows", [3, "wave", "wave + 1"])
def test_fused_rows(native, rows, cols):
    from zim_gb300 import api, synth
    if rows != 3:
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        rows = 3 * sms + sms // 4 + (rows == "wave + 1")
    ctx = api.Context(0)
    ctx.set_calibration(synth.make_rig(cols, rows, 1000.0, 100.0).as_dict(), False)
    assert (ctx.rect_h, ctx.rect_w) == (rows, cols)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(cols)
    left, right = _side(rows, cols, 8.0, gen), _side(rows, cols, 0.0, gen)
    pha_f = int(max(left[0].max(), right[0].max()))
    disp = api.rectify_match(ctx, left, right, pha_f)
    l, r = api.rectify(ctx, 0, *left, True), api.rectify(ctx, 1, *right, True)
    apart = api.match(ctx, l, r, pha_f)
    apart = apart[0] if isinstance(apart, (tuple, list)) else apart
    assert torch.equal(disp.view(torch.int32), apart.view(torch.int32))
    assert int((disp != 0).sum()) > 0 or cols < 64

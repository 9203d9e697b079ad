"""The whole-row match at widths around the rule that chooses its block size (64, 256
and 2048 columns, and all rows in one wave of the largest blocks), against itself on
a few rows at a time (the largest blocks), bit for bit; narrow windows cost less than
wide ones; and the fused rectification and match against the two apart at row counts
around one wave of its larger blocks."""
import pytest
import torch

from test_gpu_match_rows import _side

pytestmark = pytest.mark.gpu

TWO_PI = 6.283185307179586


def _row_pair(rows, cols, seed):
    """Rectified rows (base, residual, order), noisy enough for spans that are not monotone."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    out = []
    for shift in (5.0, 0.0):
        k, r = _side(rows, cols, shift, gen)
        out.append((k.contiguous(), r.contiguous(), k.contiguous()))
    return out, int(max(out[0][2].max(), out[1][2].max()))


@pytest.mark.parametrize("cols", [1, 63, 64, 65, 256, 257, 2048, 2049])
def test_block_sizes_agree(native, cols):
    from zim_gb300 import api
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = 4 * sms + 1
    ctx = api.Context(0)
    (l, r), pha_f = _row_pair(rows, cols, cols)
    disp, best = api.match(ctx, l, r, pha_f)
    for a in range(0, rows, 300):
        part = [tuple(t[a:a + 300].contiguous() for t in s) for s in (l, r)]
        d, b = api.match(ctx, part[0], part[1], pha_f)
        assert torch.equal(disp[a:a + 300].view(torch.int32), d.view(torch.int32))
        assert torch.equal(best[a:a + 300], b)
    assert int((best >= 0).sum()) > 0 or cols < 64


def _microseconds(fn):
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        fn()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            for _ in range(20):
                fn()
    torch.cuda.synchronize()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    best = float("inf")
    for _ in range(5):
        ev[0].record()
        g.replay()
        ev[1].record()
        torch.cuda.synchronize()
        best = min(best, ev[0].elapsed_time(ev[1]) * 50)
    return best


def test_narrow_windows_cost_less(native):
    """3000 rows of 64 columns against 256: three fifths of the time at most."""
    from zim_gb300 import api
    ctx = api.Context(0)
    t = []
    for cols in (64, 256):
        (l, r), pha_f = _row_pair(3000, cols, 1)
        t.append(_microseconds(lambda: api.match(ctx, l, r, pha_f, want_best=False)))
    assert t[0] <= 0.6 * t[1], t


@pytest.mark.parametrize("cols", [37, 383, 384, 385, 700])
@pytest.mark.parametrize("more", [0, 1])
def test_fused_rows_of_a_wave(native, cols, more):
    from zim_gb300 import api, synth
    rows = 4 * torch.cuda.get_device_properties(0).multi_processor_count + more
    ctx = api.Context(0)
    ctx.set_calibration(synth.make_rig(cols, rows, 1000.0, 100.0).as_dict(), False)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(cols)
    left, right = _side(rows, cols, 8.0, gen), _side(rows, cols, 0.0, gen)
    pha_f = int(max(left[0].max(), right[0].max()))
    for smooth in (False, True):
        disp = api.rectify_match(ctx, left, right, pha_f, smooth)
        l, r = api.rectify(ctx, 0, *left, smooth), api.rectify(ctx, 1, *right, smooth)
        apart, _ = api.match(ctx, l, r, pha_f)
        assert torch.equal(disp.view(torch.int32), apart.view(torch.int32))
    assert int((disp != 0).sum()) > 0 or cols < 64

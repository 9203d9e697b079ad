"""The decode's tiles: sizes around the tile (32 x 8 pixels) and the smallest image
its bulk copy takes (64 columns of 8 bits, 48 of 16, 10 rows), where frames at an odd
address (plain loads) give the copy's bits; the two sides of the rule that chooses
between strips and tiles, whose bits are the same (a pixel's result depends on its
3 x 3 neighbourhood only, so an image and its upper rows agree); and step counts and
Gray codes without code of their own, whose time per frame stays near that of those
with."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CONFIGS = [dict(encoding=0, freq=(121, 110, 120), shift_num=(8, 8, 8)),
           dict(encoding=0, freq=(121, 110, 120), shift_num=(5, 5, 5)),
           dict(encoding=1, freq=(1, 8, 64), shift_num=(4, 4, 4)),
           dict(encoding=1, freq=(1, 4, 16, 64), shift_num=(4, 4, 4, 4)),
           dict(encoding=0, freq=(121, 110, 120), shift_num=(12, 12, 12)),
           dict(encoding=3, freq=(32,), shift_num=(4,), gray_bits=5),
           dict(encoding=2, freq=(512,), shift_num=(4,), gray_bits=9)]


def _frames(cfg, rows, cols, dtype, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    full = 255 if dtype == torch.uint8 else 4095
    n = {0: 3, 1: len(cfg["freq"])}.get(cfg["encoding"], 1)
    x = torch.arange(cols, device="cuda", dtype=torch.float32)[None, :].expand(rows, cols) / cols
    out = []
    for f, steps in list(zip(cfg["freq"], cfg["shift_num"]))[:n]:
        for k in range(steps):
            out.append(0.47 + 0.35 * torch.cos(2 * np.pi * (f * x + k / steps)))
    for _ in range(cfg.get("gray_bits", 0) + (cfg["encoding"] == 3)):
        out.append(0.1 + 0.75 * (torch.rand((rows, cols), generator=g, device="cuda") < 0.5))
    f = torch.stack(out) + 0.01 * torch.randn((len(out), rows, cols), generator=g, device="cuda")
    return (f.clamp(0, 1) * full).to(torch.int32).to(dtype)


def _decode(ctx, cfg, frames):
    from zim_gb300 import api
    return api.decode(ctx, api.decode_config(**cfg, modulation_threshold=0.15), frames)


@pytest.mark.parametrize("rows,cols", [(1, 1), (7, 31), (9, 33), (10, 48), (10, 64), (9, 64), (17, 80), (24, 96)])
@pytest.mark.parametrize("dtype", [torch.uint8, torch.uint16])
@pytest.mark.parametrize("c", range(len(CONFIGS)))
def test_copy_and_plain_loads(native, c, dtype, rows, cols):
    from zim_gb300 import api
    ctx = api.Context(0)
    fr = _frames(CONFIGS[c], rows, cols, dtype, 7 * c + rows)
    odd = torch.empty(fr.numel() + 1, dtype=dtype, device="cuda")[1:].view(fr.shape)
    odd.copy_(fr)
    a, b = _decode(ctx, CONFIGS[c], fr), _decode(ctx, CONFIGS[c], odd)
    assert all(torch.equal(a[n].view(torch.uint8), b[n].view(torch.uint8)) for n in a)
    # the upper rows alone (another number of tiles): the same where all neighbours are there
    if rows > 8:
        t = _decode(ctx, CONFIGS[c], fr[:, :8].contiguous())
        assert all(torch.equal(a[n][:7].contiguous().view(torch.uint8), t[n][:7].contiguous().view(torch.uint8))
                   for n in a)
    assert ctx.check_device() == 0


@pytest.mark.parametrize("c,dtype,rows,cols", [(2, torch.uint8, 1010, 1500), (2, torch.uint16, 1010, 1500),
                                               (0, torch.uint8, 1001, 1501), (0, torch.uint16, 363, 501)])
def test_strips_and_tiles_agree(native, c, dtype, rows, cols):
    """Just above the line (strips) and, for the upper three quarters, below it (tiles)."""
    from zim_gb300 import api
    ctx = api.Context(0)
    fr = _frames(CONFIGS[c], rows, cols, dtype, c)
    part = 3 * rows // 4
    a, t = _decode(ctx, CONFIGS[c], fr), _decode(ctx, CONFIGS[c], fr[:, :part].contiguous())
    for n in a:
        assert torch.equal(a[n][:part - 1].contiguous().view(torch.uint8), t[n][:part - 1].contiguous().view(torch.uint8))
    assert float(a["valid"].float().mean()) > 0.9


def _microseconds(fn):
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    best = float("inf")
    for _ in range(5):
        ev[0].record()
        for _ in range(20):
            fn()
        ev[1].record()
        torch.cuda.synchronize()
        best = min(best, ev[0].elapsed_time(ev[1]) * 50)
    return best


@pytest.mark.parametrize("few,many,dtype,factor", [(1, 0, torch.uint8, 1.5), (1, 0, torch.uint16, 1.5),
                                                   (6, 5, torch.uint8, 1.5 * 13 / 10), (6, 5, torch.uint16, 1.5 * 13 / 10)])
def test_other_step_counts_keep_up(native, few, many, dtype, factor):
    """15 frames (five steps) against 24 (eight), and 13 frames of a nine-bit Gray code
    against the 10 of a five-bit one, at 2448 x 2048: half as much again at most."""
    from zim_gb300 import api
    ctx = api.Context(0)
    t = []
    for c in (few, many):
        fr = _frames(CONFIGS[c], 2048, 2448, dtype, c)
        t.append(_microseconds(lambda: _decode(ctx, CONFIGS[c], fr)))
    assert t[0] <= factor * t[1], t


@pytest.mark.parametrize("dtype", [torch.uint8, torch.uint16])
def test_hdr_step_counts_keep_up(native, dtype):
    """36 HDR frames (twelve steps, no code of their own) against 24 (eight) at 2448 x
    2048: the frames' ratio and half as much again at most."""
    from zim_gb300 import api
    ctx = api.Context(0)
    t = []
    for c in (4, 0):
        cfg = dict(CONFIGS[c], enable_hdr=True, hdr_saturation_gray=200.0 if dtype == torch.uint8 else 3200.0)
        fr = _frames(cfg, 2048, 2448, dtype, c)
        t.append(_microseconds(lambda: _decode(ctx, cfg, fr)))
    assert t[0] <= 1.5 * 36 / 24 * t[1], t

"""The decode at image sizes around its strips (30 columns per warp, bands of 4 to
32 rows) and for every step count and encoding it has its own code for, against
the FP64 oracle on noisy fringes: orders and validity equal except where the
oracle flags a decision within 1e-5 of its threshold, phases within 1e-5 rad (the
decode's stated tolerance)."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CONFIGS = [dict(encoding=0, freq=(121, 110, 120), shift_num=(8, 8, 8)),
           dict(encoding=0, freq=(107, 100, 94), shift_num=(4, 4, 4), avg_three_phase=False),
           dict(encoding=1, freq=(1, 8, 64), shift_num=(4, 4, 4)),
           dict(encoding=1, freq=(1, 4, 16, 64), shift_num=(3, 5, 4, 9)),
           dict(encoding=2, freq=(32,), shift_num=(4,), gray_bits=5),
           dict(encoding=3, freq=(32,), shift_num=(6,), gray_bits=8),
           dict(encoding=0, freq=(121, 110, 120), shift_num=(8, 8, 8), enable_hdr=True),
           dict(encoding=1, freq=(1, 8, 64), shift_num=(4, 7, 4), enable_hdr=True)]
SIZES = [(1, 1), (3, 29), (5, 30), (4, 31), (33, 61), (70, 122)]


def _frames(cfg, rows, cols, bits, seed):
    """Fringes of the configuration's frequencies across the image, noise, dark and saturated patches."""
    g = np.random.default_rng(seed)
    top = 255 if bits == 8 else 4095
    u = (np.arange(cols) + 0.5)[None, :] / cols * np.ones((rows, 1)) + g.normal(0, 1e-4, (rows, cols))
    A, B = top * g.uniform(0.35, 0.5, (rows, cols)), top * g.uniform(0.2, 0.35, (rows, cols))
    B[g.random((rows, cols)) < 0.1] = 0
    n = len(cfg["freq"]) if cfg["encoding"] != 0 else 3
    n = 1 if cfg["encoding"] >= 2 else n
    out = []
    for i in range(n):
        for k in range(cfg["shift_num"][i]):
            out.append(A + B * np.cos(2 * math.pi * cfg["freq"][i] * u + 2 * math.pi * k / cfg["shift_num"][i]))
    for _ in range(cfg.get("gray_bits", 0) + (cfg["encoding"] == 3)):
        out.append(A + B * np.where(g.random((rows, cols)) < 0.5, 1, -1))
    f = np.stack(out) + g.normal(0, top / 120, (len(out), rows, cols))
    if cfg.get("enable_hdr"):
        f *= 1.25
    return np.clip(np.rint(f), 0, top).astype(np.uint8 if bits == 8 else np.uint16)


@pytest.mark.parametrize("rows,cols", SIZES)
@pytest.mark.parametrize("bits", [8, 12])
@pytest.mark.parametrize("c", range(len(CONFIGS)))
def test_decode_strip_edges(ctx, oracle_lib, c, bits, rows, cols):
    from zim_gb300 import api
    import oracle
    kw = dict(CONFIGS[c], modulation_threshold=0.15)
    if kw.get("enable_hdr"):
        kw.update(hdr_saturation_gray=255.0 if bits == 8 else 4095.0, hdr_min_amplitude=2.0 if bits == 8 else 32.0)
    fr = _frames(kw, rows, cols, bits, 100 * c + rows)
    d = api.decode(ctx, api.decode_config(**kw), torch.from_numpy(fr).cuda())
    ph, k, mod, valid, near = oracle.decode(oracle.make_decode_cfg(**kw), fr)
    gk, gv = d["order"].cpu().numpy(), d["valid"].cpu().numpy()
    assert (((gk != k) | (gv != valid)) & (near == 0)).sum() == 0
    ok = (valid > 0) & (gv > 0) & (near == 0) & (gk == k)
    err = np.abs(d["residual"].cpu().numpy().astype(np.float64) - (ph - 2 * math.pi * k))[ok]
    assert err.size == 0 or err.max() <= 1e-5
    # frames at an odd address: the unaligned loads give the same bits
    t = torch.from_numpy(fr).cuda()
    odd = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape)
    odd.copy_(t)
    e = api.decode(ctx, api.decode_config(**kw), odd)
    assert all(torch.equal(d[n], e[n]) for n in d)

"""A pair's cameras decoded and smoothed in one launch against each camera in a
launch of its own: the whole pair's disparity against decode, rectification and
match, and median apart, bit for bit, for every decode kernel, at widths that are
no multiple of the strips and with right frames off the left ones' alignment."""
import numpy as np
import pytest
import torch

from conftest import scene_data

pytestmark = pytest.mark.gpu


def _offset(t):
    """The same frames one sample off their alignment."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")
    buf[1:] = t.reshape(-1)
    return buf[1:].reshape(t.shape)


@pytest.mark.parametrize("off", [False, True])
@pytest.mark.parametrize("name,hdr", [("config0", False), ("config1", False), ("ref_heterodyne", False),
                                      ("ref_heterodyne", True)])
@pytest.mark.parametrize("width,height", [(31, 33), (182, 97)])
def test_pair_equals_single_cameras(native, name, hdr, off, width, height):
    from zim_gb300 import api
    spec, left, right, _ = scene_data(name, width=width, height=height)
    L, R = torch.from_numpy(np.ascontiguousarray(left)).cuda(), torch.from_numpy(np.ascontiguousarray(right)).cuda()
    if off:
        R = _offset(R)
    ctx = api.Context(0)
    ctx.set_calibration(spec.rig.as_dict(), True)
    kw = spec.decode_kwargs()
    if hdr:
        kw.update(enable_hdr=True, hdr_saturation_gray=255.0, hdr_min_amplitude=2.0)
    dcfg = api.decode_config(**kw)
    rcfg = api.recon_config(use_px_gaussian=0, use_ror=0)
    _, _, disp = api.reconstruct_pair(ctx, dcfg, rcfg, L, R, spec.pha_f, want_disp=True)
    one = [api.decode(ctx, dcfg, f) for f in (L, R)]
    raw = api.rectify_match(ctx, *[(o["order"], o["residual"]) for o in one], spec.pha_f, hdr=hdr)
    med = api.median_reproject(ctx, rcfg, raw)[0]
    assert torch.equal(disp.view(torch.int32), med.view(torch.int32))

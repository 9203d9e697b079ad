"""The launches that a batch replay counts: every pair more of the same kind adds one
decode launch (both cameras), the other stages are the batch's."""
import pytest
import torch

from conftest import scene_data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [{}, {"use_sor": 1, "sor_mean_k": 20}])
def test_launches_per_replay(native, kw):
    from zim_gb300 import api
    from zim_gb300.batch import Batch, BatchPair
    spec, L, R, _ = scene_data("config0")
    dcfg = api.decode_config(**spec.decode_kwargs())
    rcfg = api.recon_config(**kw)
    ctx = api.Context(0)
    ctx.set_calibration(spec.rig.as_dict(), True)
    left, right = torch.from_numpy(L).cuda(), torch.from_numpy(R).cuda()
    counts = []
    for n in (1, 2, 5):
        b = Batch(ctx, [spec.rig.as_dict()])
        b.submit([BatchPair(dcfg, left, right) for _ in range(n)], rcfg)
        before = ctx.launch_count()
        b.run()
        b.run()
        counts.append((ctx.launch_count() - before) / 2)
        b.close()
    # SOR with pixel rays: tree, window, search, statistics, classification per pair
    per_pair = 1 + (5 if kw else 0)
    assert counts[1] - counts[0] == per_pair and counts[2] - counts[0] == 4 * per_pair

"""The radius filter at window sizes around the line between rings alone and rings
followed by rows, and at cloud sizes around the rules for a tile's rows, against the
definition: the coordinates are small integers, so every squared distance is exact.
Where nobody has enough neighbours, a wide window costs about what its pixels do."""
import pytest
import torch

from test_gpu_match_windows import _microseconds

pytestmark = pytest.mark.gpu


def _cloud(rows, cols, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    y, x = torch.meshgrid(torch.arange(rows, device="cuda"), torch.arange(cols, device="cuda"), indexing="ij")
    z = torch.randint(0, 6, (rows, cols), generator=g, device="cuda")
    xyz = torch.stack([x, y, z], -1).float()
    mask = (torch.rand((rows, cols), generator=g, device="cuda") < 0.7).to(torch.uint8)
    return xyz, mask


def _expected(xyz, mask, r2, min_nb, hw):
    rows, cols = mask.shape
    n = torch.zeros((rows, cols), dtype=torch.int32, device="cuda")
    for dy in range(-hw, hw + 1):
        for dx in range(-hw, hw + 1):
            ys, xs = slice(max(0, -dy), min(rows, rows - dy)), slice(max(0, -dx), min(cols, cols - dx))
            yt, xt = slice(max(0, dy), min(rows, rows + dy)), slice(max(0, dx), min(cols, cols + dx))
            if (dy == 0 and dx == 0) or ys.stop <= ys.start or xs.stop <= xs.start:
                continue
            d2 = ((xyz[ys, xs] - xyz[yt, xt]) ** 2).sum(-1)
            n[ys, xs] += ((d2 <= r2) & (mask[yt, xt] > 0)).int()
    return ((mask > 0) & (n >= min_nb)).to(torch.uint8)


@pytest.mark.parametrize("window", [0, 2, 20, 21, 22, 23, 40, 96])
@pytest.mark.parametrize("rows,cols", [(1, 40), (33, 65), (70, 31)])
def test_windows_against_the_definition(native, rows, cols, window):
    from zim_gb300 import api
    ctx = api.Context(0)
    xyz, mask = _cloud(rows, cols, window)
    for radius, min_nb in ((2.9, 4), (6.5, 40), (9.3, 110), (12.4, 250), (40.2, 900)):
        out, mo = api.filter_ror(ctx, xyz, mask, radius, min_nb, window)
        ref = _expected(xyz, mask, float(torch.tensor(radius, dtype=torch.float32) ** 2), min_nb, window // 2)
        assert torch.equal(mo, ref)
        assert torch.equal(out, xyz * ref[..., None])


@pytest.mark.parametrize("rows,cols", [(480, 640), (873, 1101), (1100, 1400)])
def test_tile_rows_agree(native, rows, cols):
    from zim_gb300 import api
    ctx = api.Context(0)
    xyz, mask = _cloud(rows, cols, 3)
    out, mo = api.filter_ror(ctx, xyz, mask, 3.2, 9, 10)
    assert torch.equal(mo, _expected(xyz, mask, 3.2 ** 2, 9, 5)) and 0.1 < mo.float().mean() < 0.69
    assert torch.equal(out, xyz * mo[..., None])


def test_wide_windows_without_neighbours(native):
    """A 91 x 91 window has 4.9 times the pixels of a 41 x 41 one: 7.2 times the time at most."""
    from zim_gb300 import api
    ctx = api.Context(0)
    xyz, mask = _cloud(768, 1024, 5)
    t = [_microseconds(lambda: api.filter_ror(ctx, xyz, mask, 0.1, 10, w)) for w in (40, 90)]
    assert t[1] <= 7.2 * t[0], t


@pytest.mark.parametrize("window", [4, 30])
@pytest.mark.parametrize("radius", [7.5, 1e20])
def test_points_without_finite_coordinates(native, window, radius):
    """The definition as the reference counts: float distances over the window, the point's
    own among them, at least min_nb + 1 (any with min_nb 0).  A point without finite
    coordinates does not count itself, and with a radius whose square is infinite one at
    infinity has the finite ones near."""
    from zim_gb300 import api
    ctx = api.Context(0)
    xyz = torch.arange(3 * 25, device="cuda", dtype=torch.float32).view(5, 5, 3)
    mask = torch.ones((5, 5), dtype=torch.uint8, device="cuda")
    xyz[2, 2, 0], xyz[0, 0] = float("inf"), float("nan")
    p, r = xyz.view(25, 3), torch.tensor(radius, dtype=torch.float32, device="cuda")
    y, x = torch.arange(25, device="cuda") // 5, torch.arange(25, device="cuda") % 5
    near = ((y[:, None] - y).abs() <= window // 2) & ((x[:, None] - x).abs() <= window // 2)
    count = ((((p[:, None] - p) ** 2).sum(-1) <= r * r) & near).sum(1).view(5, 5)
    for min_nb in (0, 1, 2, 8, 14, 22, 23, 24):
        _, mo = api.filter_ror(ctx, xyz, mask, radius, min_nb, window)
        want = (count >= min_nb + 1) | (min_nb == 0)
        assert torch.equal(mo, want.to(torch.uint8)), min_nb

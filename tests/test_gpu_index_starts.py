"""Bin starts filled by the gather (up to 2^16 bins) and by searches: the line
between them, a single bin, gaps of one bin to all of them, and the counts
around a block and a warp of records.  The pairs that the density scans have to
be all pairs within 3h."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["uniform", "corners"])
@pytest.mark.parametrize("bins", [1, 2, 31, 256, 257])  # per side
@pytest.mark.parametrize("n", [1, 31, 256, 257, 5000])
def test_bin_starts(n, bins, kind):
    r = np.random.default_rng(n + bins)
    top = bins - 0.5
    x, y = r.uniform(0, top, n), r.uniform(0, top, n)
    if kind == "corners":
        x, y = top * (x > top / 2), top * (y > top / 2)
    x[0], y[0], x[-1], y[-1] = 0.0, 0.0, top, top  # the extent is [0, top] squared
    x, y = (torch.from_numpy(a.astype(np.float32)).cuda() for a in (x, y))
    h = max(0.35, bins / 40.0)
    g = mk.Grid(33, 33, -0.5, -0.5, (top + 1.0) / 33)
    torch.cuda.synchronize()
    with mk.Context(0) as ctx:
        pts = mk.Points.wrap(ctx, x, y, None)
        mk.unit_edge_weights(ctx, pts)
        idx = mk.Index(ctx, pts, h, 1.0)
        out = torch.empty(33, 33, device="cuda")
        pairs = mk.density_tile(ctx, idx, g, 0, 0, 33, 33, None, out, count=True)
    cs, org = (float(np.float32(v)) for v in (g.cs, g.xll))
    c = (org + (torch.arange(33, device="cuda", dtype=torch.float64) + 0.5) * cs).float().double()
    d2 = (c[None, :, None] - x.double()) ** 2 + (c[:, None, None] - y.double()) ** 2
    assert pairs == int((d2 < 9.0 * float(np.float32(h) * np.float32(h))).sum())

"""An index under a budget of its points, its own arrays, three buffers of a
word a point (the sort's keys and values) and 64 KB: built, and the same as an
unlimited one (a tile's density, bit for bit)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


def held(b):  # bytes the context holds for a block of b
    if b > 1 << 20:
        return -(-b // (2 << 20)) * (2 << 20)
    return max(256, 1 << (int(b) - 1).bit_length())


@pytest.mark.parametrize("h", [0.1, 2.0, 40.0])  # the largest bin grid (4,097^2: three 9-bit digits), ordinary ones
@pytest.mark.parametrize("n", [90, 700, 5000, 20_000, 60_000, 70_000])
def test_index_budget(n, h):
    r = np.random.default_rng(n)
    x, y = r.uniform(0, 1000, n).astype(np.float32), r.uniform(0, 1000, n).astype(np.float32)
    ex, ey = float(x.max()) - float(x.min()), float(y.max()) - float(y.min())
    side = max(0.5 * h, max(ex, ey) / 4096)
    nbins = (int(ex / side) + 1) * (int(ey / side) + 1)
    budget = 3 * held(4 * n) + held(8 * n)  # x, y, edge weights, distances
    budget += held(4 * (nbins + 1)) + held(32 * n) + held(4 * n) + 3 * held(4 * n) + (64 << 10)
    g = mk.Grid(1000, 1000, 0.0, 0.0, 1.0, -9999.0)
    res = []
    for b in (0, budget):
        with mk.Context(0, hbm_budget=b) as ctx:
            pts = mk.Points.upload(ctx, x, y)
            mk.unit_edge_weights(ctx, pts)
            idx = mk.Index(ctx, pts, h)
            out = torch.empty(32, 32, device="cuda")
            if h < 10.0:  # few candidates: no split, no scratch
                torch.cuda.synchronize()
                mk.density_tile(ctx, idx, g, 500, 300, 32, 32, None, out)
                res.append(out)
    assert not res or torch.equal(res[0], res[1])

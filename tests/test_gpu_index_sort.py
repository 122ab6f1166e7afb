"""The index build at the sizes where its sort can go wrong: counts around a
tile of 256, 1,024 and 4,096 items, one to three digit passes, many points in
one bin and most bins empty.  Every point has to be found in the right bins:
densities on a coarse raster against FP64 sums over all points (1e-6
relative, exactly 0 where no point is in reach), and the leave-one-out pair
count (whose query order is a second sort) against all pairs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


def points(n, kind):
    r = np.random.default_rng(n)
    x, y = r.uniform(0, 1000, n), r.uniform(0, 1000, n)
    if kind == "knot" and n > 2:  # all but two corner points in one spot
        x[:-2], y[:-2] = 512.5 + r.uniform(-1e-3, 1e-3, n - 2), 487.5 + r.uniform(-1e-3, 1e-3, n - 2)
        x[-2:], y[-2:] = [0, 1000], [0, 1000]
    return tuple(torch.from_numpy(a.astype(np.float32)).cuda() for a in (x, y, r.lognormal(0, 0.5, n)))


@pytest.mark.parametrize("kind", ["uniform", "knot"])
@pytest.mark.parametrize("h", [400.0, 20.0, 0.4])
@pytest.mark.parametrize("n", [1, 255, 257, 4097, 65535, 65537, 524_289])
def test_index_holds_every_point_once(n, h, kind):
    x, y, w = points(n, kind)
    g = mk.Grid(40, 40, 0.0, 0.0, 25.0)
    torch.cuda.synchronize()
    with mk.Context(0) as ctx:
        pts = mk.Points.wrap(ctx, x, y, w)
        mk.unit_edge_weights(ctx, pts)
        idx = mk.Index(ctx, pts, h)
        out = torch.empty(40, 40, device="cuda")
        pairs = mk.density_tile(ctx, idx, g, 0, 0, 40, 40, None, out, count=True)
        got = out.double()
    h2 = float(np.float32(h) * np.float32(h))
    cx = (torch.arange(40, device="cuda", dtype=torch.float64) + 0.5) * 25.0
    ref, count = torch.zeros(40, 40, device="cuda", dtype=torch.float64), 0
    for r in range(40):
        dy2 = (cx[39 - r] - y.double()) ** 2
        d2 = (cx[:, None] - x.double()[None, :]) ** 2 + dy2[None, :]
        inside = d2 < 9.0 * h2
        count += int(inside.sum())
        ref[r] = (torch.exp(d2 / (-2.0 * h2)) * inside * w.double()[None, :]).sum(1)
    ref /= h2 * float(np.float32(2 * np.pi))
    assert pairs == count
    assert torch.equal(got == 0, ref == 0)
    assert float(((got - ref).abs() / ref.clamp_min(1e-300)).max()) <= 1e-6


@pytest.mark.parametrize("n", [2, 257, 4097, 70_001])
def test_query_order_holds_every_point_once(n):
    x, y, w = points(n, "uniform")
    torch.cuda.synchronize()
    h = 1000.0 / n ** 0.5
    with mk.Context(0) as ctx:
        pts = mk.Points.wrap(ctx, x, y, w)
        mk.log_likelihood_batch(ctx, pts, None, [h])
        pairs = ctx.last_loo_evals[1]
    h2, count = float(np.float32(h) * np.float32(h)), 0
    for p in range(0, n, 2048):
        d2 = (x[p:p + 2048, None].double() - x.double()) ** 2 + (y[p:p + 2048, None].double() - y.double()) ** 2
        count += int((d2 < 9.0 * h2).sum())
    assert pairs == count - n

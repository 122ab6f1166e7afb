"""The adaptive likelihood at every budget: an error, or the unlimited answer
(the queries' order and the split of their windows are given up first), and no
error once the budget holds the points, an index of them, the sort's buffers
and one partial sum per point and split in eight."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


def mixture(n):
    r = np.random.default_rng(n)
    c = r.uniform(300, 1700, (12, 2))
    xy = np.clip(c[r.integers(0, 12, n)] + r.normal(0, 120, (n, 2)), 20, 1980).astype(np.float32)
    return xy[:, 0].copy(), xy[:, 1].copy(), r.uniform(0.5, 2, n).astype(np.float32)


def likelihood(ctx, x, y, w, g, m):
    pts = mk.Points.upload(ctx, x, y, w)
    ras = mk.Raster.upload(ctx, g, m)
    mk.calc_dist2_boundary(ctx, pts, ras)
    return mk.loglik_adaptive(ctx, pts, ras, 40.0, -0.5)


@pytest.mark.parametrize("n,enough", [(3000, 1700), (20_000, 6100), (200_000, 26_800)])
def test_every_budget(n, enough):
    x, y, w = mixture(n)
    yy, xx = np.mgrid[0:200, 0:200] - 99.5
    m = np.where(np.hypot(xx, yy) < 98.0, 1.0, -9999.0).astype(np.float32)
    g = mk.Grid(200, 200, 0.0, 0.0, 10.0, -9999.0)
    with mk.Context(0) as ctx:
        ref = likelihood(ctx, x, y, w, g, m)
    fits = 0
    for kib in np.linspace(0.4 * enough, 2.0 * enough, 33).astype(int):
        with mk.Context(0, hbm_budget=int(kib) << 10) as ctx:
            try:
                got = likelihood(ctx, x, y, w, g, m)
            except mk.MgkError as e:
                assert e.status == -3 and kib < enough
                continue
            fits += 1
            assert abs(got - ref) <= 1e-8 * abs(ref)
    assert fits >= 10

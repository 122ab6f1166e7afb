"""One bandwidth with edge correction under budgets that hold what the batch
needs but not what only speeds it up (the weights in record order, 0.8 MB here):
accepted, with the unlimited answer (the parity tests' tolerance)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


def score(ctx, x, y, w, g, m):
    pts = mk.Points.upload(ctx, x, y, w)
    ras = mk.Raster.upload(ctx, g, m)
    mk.calc_dist2_boundary(ctx, pts, ras)
    return mk.log_likelihood_batch(ctx, pts, ras, np.array([8.0], np.float32))[0][0]


def test_one_bandwidth():
    n = 200_000
    r = np.random.default_rng(1)
    c = r.uniform(300, 1700, (12, 2))
    xy = np.clip(c[r.integers(0, 12, n)] + r.normal(0, 120, (n, 2)), 20, 1980).astype(np.float32)
    x, y, w = xy[:, 0].copy(), xy[:, 1].copy(), r.uniform(0.5, 2, n).astype(np.float32)
    yy, xx = np.mgrid[0:200, 0:200] - 99.5
    m = np.where(np.hypot(xx, yy) < 98.0, 1.0, -9999.0).astype(np.float32)
    g = mk.Grid(200, 200, 0.0, 0.0, 10.0, -9999.0)
    with mk.Context(0) as ctx:
        ref = score(ctx, x, y, w, g, m)
    for kib in range(21_500, 26_000, 250):
        with mk.Context(0, hbm_budget=kib << 10) as ctx:
            assert abs(score(ctx, x, y, w, g, m) - ref) <= 1e-6 * abs(ref)

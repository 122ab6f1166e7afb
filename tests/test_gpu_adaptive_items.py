"""The adaptive likelihood's point densities at the sizes where their work
items can go wrong: counts around a warp of queries (32), windows of more
runs of bins than one table holds (64), narrow and wide bandwidths side by
side.  Against the FP64 oracle at the parity tests' tolerance (1e-6 relative
+ 1e-6)."""
import numpy as np
import pytest

import oracle_py as o

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mask", [False, True])
@pytest.mark.parametrize("n,h", [(2, 30.0), (31, 8.0), (33, 8.0), (97, 20.0), (700, 3.0), (4000, 12.0)])
def test_adaptive_likelihood_items(n, h, mask):
    r = np.random.default_rng(n)
    k = n // 2  # a dense knot (narrow bandwidths) in a sparse field (wide ones)
    x = np.concatenate([r.normal(150.0, 2.0, k), r.uniform(0, 400, n - k)]).astype(np.float32)
    y = np.concatenate([r.normal(220.0, 2.0, k), r.uniform(0, 400, n - k)]).astype(np.float32)
    w = r.lognormal(0, 0.5, n).astype(np.float32)
    g = em = d2 = None
    with mk.Context(0) as ctx:
        pts, ras = mk.Points.upload(ctx, x, y, w), None
        if mask:
            g = o.grid(50, 50, 0.0, 0.0, 8.0, -9999.0)
            em = np.where(np.hypot(*(np.mgrid[0:50, 0:50] - 25.0)) < 23.0, 1.0, -9999.0).astype(np.float32)
            d2 = o.dist2_boundary(x, y, g, o.mark_boundary(g, em))
            ras = mk.Raster.upload(ctx, mk.Grid.of(g), em)
            mk.calc_dist2_boundary(ctx, pts, ras)
        for alpha in (-0.5, -0.2):
            ref, _ = o.loglik_adaptive(x, y, w, d2, g, em, h, alpha)
            got = mk.loglik_adaptive(ctx, pts, ras, h, alpha)
            assert abs(got - ref) <= 1e-6 * abs(ref) + 1e-6
            assert got == mk.loglik_adaptive(ctx, pts, ras, h, alpha)

"""Bandwidth lists longer than a launch grid's second dimension (65,535)."""
import numpy as np
import pytest

import oracle_py as o

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edge", [False, True])
def test_list_of_70_000(edge):
    r = np.random.default_rng(4)
    n = 140
    x, y = r.uniform(0, 60, n).astype(np.float32), r.uniform(0, 60, n).astype(np.float32)
    few = np.array([0.5, 1.0, 2.5, 4.0, 6.0, 9.0, 14.0], np.float32)
    hs = np.tile(few, 10_000)
    g = o.grid(30, 30, 0.0, 0.0, 2.0, -9999.0)
    m = np.ones((30, 30), np.float32)
    d2 = o.dist2_boundary(x, y, g, o.mark_boundary(g, m))
    w = np.ones(n, np.float32)
    ref = np.array([o.loglik_at(x, y, w, d2, g, m, float(h))[0] if edge else o.loo_loglik(x, y, w, None, float(h))[0]
                    for h in few])
    with mk.Context(0) as ctx:
        pts, ras = mk.Points.upload(ctx, x, y), None
        if edge:
            ras = mk.Raster.upload(ctx, mk.Grid.of(g), m)
            mk.calc_dist2_boundary(ctx, pts, ras)
        got, best = mk.log_likelihood_batch(ctx, pts, ras, hs)
    assert np.all(np.abs(got - np.tile(ref, 10_000)) <= np.tile(1e-6 * np.abs(ref) + 1e-6, 10_000))
    assert best == int(np.argmax(got)) < len(few)

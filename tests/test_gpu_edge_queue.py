"""Edge weights of lists that a counter hands out to the warps (about 14,000
points near the boundary and more) against the same points in short lists,
which it does not: each weight depends on its point alone, so they are equal
bit for bit, for one wide bandwidth and for per-point ones."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("varh", [False, True])
@pytest.mark.parametrize("n", [13_000, 14_300, 29_001, 60_000])
def test_long_lists_equal_short_ones(n, varh):
    r = np.random.default_rng(n)
    x, y = (torch.from_numpy(r.uniform(0, 400, n).astype(np.float32)).cuda() for _ in range(2))
    hp = torch.from_numpy((30.0 * np.exp(0.7 * r.standard_normal(n))).astype(np.float32)).cuda() if varh else None
    g = mk.Grid(100, 90, 0.0, 20.0, 4.0, -9999.0)
    yy, xx = np.mgrid[0:90, 0:100]
    mask = np.where(np.hypot(xx - 50.0, yy - 45.0) < 44.0 + 4 * np.sin(xx), 1.0, -9999.0).astype(np.float32)
    h = 0.0 if varh else 150.0  # every point lies within 3h of the boundary
    torch.cuda.synchronize()
    with mk.Context(0) as ctx:
        ras = mk.Raster.upload(ctx, g, mask)
        mk.mark_boundary(ctx, ras)

        def weights(a, b):
            part = [v[a:b].clone() if v is not None else None for v in (x, y, None, hp)]
            pts = mk.Points.wrap(ctx, *part)
            torch.cuda.synchronize()
            mk.calc_dist2_boundary(ctx, pts, ras)
            mk.edge_correction_weights(ctx, pts, ras, h)
            return pts.download(ew=True)[1]

        whole = weights(0, n)
        parts = np.concatenate([weights(a, min(n, a + 2000)) for a in range(0, n, 2000)])
    assert np.array_equal(whole, parts)

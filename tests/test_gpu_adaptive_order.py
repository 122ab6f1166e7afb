"""The adaptive likelihood's query order on both sides of the count from which
it follows a curve (8,192): clustered and uniform points, all points in one
spot (an extent of zero), and all on a line.  Against the FP64 oracle at the
parity tests' tolerance (1e-6 relative + 1e-6)."""
import numpy as np
import pytest

import oracle_py as o

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kind", [(8191, "clusters"), (8192, "clusters"), (8225, "uniform"), (8192, "spot"), (8193, "line")])
def test_adaptive_likelihood_order(n, kind):
    r = np.random.default_rng(n)
    if kind == "clusters":
        c = r.uniform(100, 900, (8, 2))
        xy = c[r.integers(0, 8, n)] + 25.0 * r.standard_normal((n, 2))
    else:
        xy = r.uniform(0, 1000, (n, 2))
    if kind == "spot":
        xy[:] = 321.25, 45.5
    if kind == "line":
        xy[:, 1] = 7.0
    x, y = xy.astype(np.float32).T.copy()
    w = r.lognormal(0, 0.5, n).astype(np.float32)
    with mk.Context(0) as ctx:
        pts = mk.Points.upload(ctx, x, y, w)
        ref, _ = o.loglik_adaptive(x, y, w, None, None, None, 6.0, -0.5)
        got = mk.loglik_adaptive(ctx, pts, None, 6.0, -0.5)
        assert abs(got - ref) <= 1e-6 * abs(ref) + 1e-6
        assert got == mk.loglik_adaptive(ctx, pts, None, 6.0, -0.5)

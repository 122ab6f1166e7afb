"""The point scans at bandwidths where a product of the exponent's parts, or the
cutoff itself, leaves FP32: the slots past a window's candidates must stay
outside for every h.  Against the FP64 oracle (adaptive 1e-8 relative, as the
search's parity test holds it; the batch 1e-6 relative + 1e-6), pair counts
equal."""
import numpy as np
import pytest

import oracle_py as o

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


def points(n):
    """On a line, two of them in one place from 33 points."""
    r = np.random.default_rng(n)
    x, y = r.uniform(0, 570, n).astype(np.float32), np.full(n, 287.25, np.float32)
    if n >= 33:
        x[5] = x[20]
    return x, y, np.ones(n, np.float32)


@pytest.mark.parametrize("n", [1, 31, 33, 70])
@pytest.mark.parametrize("h", [1e-15, 1e-9, 2.861023e-06, 1e-5, 1e-3])
def test_far_below_the_points_spacing(n, h):
    x, y, w = points(n)
    with mk.Context(0) as ctx:
        pts = mk.Points.upload(ctx, x, y, w)
        got = mk.loglik_adaptive(ctx, pts, None, h, -1.0)
        pairs = ctx.last_loo_evals[1]
        ref, _ = o.loglik_adaptive(x, y, w, None, None, None, float(np.float32(h)), -1.0)
        # the pilot's pairs (every point with itself) and the leave-one-out ones
        assert abs(got - ref) <= 1e-8 * abs(ref) and pairs == n + 2 * (2 if n >= 33 else 0)
        ll, _ = mk.log_likelihood_batch(ctx, pts, None, np.array([h], np.float32))
        lref, _, levals = o.loo_loglik(x, y, w, None, float(np.float32(h)))
        assert abs(ll[0] - lref) <= 1e-6 * abs(lref) + 1e-6 and ctx.last_loo_evals[1] == levals


@pytest.mark.parametrize("n", [1, 31, 33, 70])
@pytest.mark.parametrize("h", [1e17, 3.3333e17, 4e18, 7e18, 1.5e19])
def test_far_above_the_points_extent(n, h):
    """Every pair counts; every density is below its floor."""
    x, y, w = points(n)
    floor = n * np.log(float(np.float32(1e-14)))
    with mk.Context(0) as ctx:
        pts = mk.Points.upload(ctx, x, y, w)
        ll, _ = mk.log_likelihood_batch(ctx, pts, None, np.array([h], np.float32))
        assert abs(ll[0] - floor) <= 1e-8 * abs(floor) and ctx.last_loo_evals[1] == n * (n - 1)
        got = mk.loglik_adaptive(ctx, pts, None, h, -0.5)
        assert abs(got - floor) <= 1e-8 * abs(floor) and ctx.last_loo_evals[1] == n * n + n * (n - 1)

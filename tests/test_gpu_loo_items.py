"""The leave-one-out scan at the sizes where its work items can go wrong:
counts around a query group (128) and a quarter of one (32), windows of more
bin rows than one stretch (32) with empty stretches among them, groups split
into parts, clusters denser than a Kahan piece, far coordinates, and budgets
too small for the weights in record order.  Against the FP64 oracle, at the
parity tests' tolerance (1e-6 relative + 1e-6), pair counts equal."""
import numpy as np
import pytest

import oracle_py as o

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


def points(n, kind, seed):
    r = np.random.default_rng(seed)
    if kind == "clustered":  # a dense knot and a sparse rest: long windows, empty bin rows
        k = n // 2
        x = np.concatenate([r.normal(40.0, 0.5, k), r.uniform(0, 400, n - k)])
        y = np.concatenate([r.normal(350.0, 0.5, k), r.uniform(0, 400, n - k)])
    else:
        x, y = r.uniform(0, 60, n), r.uniform(0, 60, n)
    off = 39_620.0 if kind == "far" else 0.0
    return (x + off).astype(np.float32), (y + off).astype(np.float32), r.lognormal(0, 0.5, n).astype(np.float32)


def disc_mask(g):
    yy, xx = np.mgrid[0:g.nrows, 0:g.ncols]
    inside = (xx - g.ncols / 2) ** 2 + (yy - g.nrows / 2) ** 2 < (0.45 * g.ncols) ** 2
    return np.where(inside, 1.0, g.nodata).astype(np.float32)


def run(ctx, x, y, w, hgrid, eg, em):
    pts = mk.Points.upload(ctx, x, y, w)
    ras = None
    if em is not None:
        ras = mk.Raster.upload(ctx, mk.Grid.of(eg), em)
        mk.calc_dist2_boundary(ctx, pts, ras)
    logl, best = mk.log_likelihood_batch(ctx, pts, ras, hgrid)
    return logl, best, ctx.last_loo_evals


def reference(x, y, w, hgrid, eg, em):
    if em is None:
        r = [o.loo_loglik(x, y, w, None, float(h)) for h in hgrid]
        return np.array([v[0] for v in r]), sum(v[2] for v in r)
    d2 = o.dist2_boundary(x, y, eg, o.mark_boundary(eg, em))
    r = [o.loglik_at(x, y, w, d2, eg, em, float(h)) for h in hgrid]
    return np.array([v[0] for v in r]), sum(v[1] for v in r)


@pytest.mark.parametrize("kind", ["uniform", "clustered", "far"])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 127, 129, 700, 5000])
def test_loo_items(n, kind):
    x, y, w = points(n, kind, n)
    hgrid = np.array([0.3, 0.9, 2.5, 7.0, 20.0], np.float32)
    eg = o.grid(50, 50, 39_620.0 if kind == "far" else 0.0, 39_620.0 if kind == "far" else 0.0,
                8.0 if kind == "clustered" else 1.2, -9999.0)
    em = None if n % 2 else disc_mask(eg)
    ref, evals = reference(x, y, w, hgrid, eg, em)
    with mk.Context(0) as ctx:
        got, best, ev = run(ctx, x, y, w, hgrid, eg, em)
        assert np.all(np.abs(got - ref) <= 1e-6 * np.abs(ref) + 1e-6)
        assert best == int(np.argmax(got)) and sum(ev) == evals
        again, _, _ = run(ctx, x, y, w, hgrid, eg, em)
        assert np.array_equal(got.view(np.uint64), again.view(np.uint64))


def test_loo_under_small_budgets():
    """At every budget the call either says so or gives the same answer."""
    x, y, w = points(20_000, "uniform", 3)
    hgrid = np.linspace(1.0, 4.0, 24).astype(np.float32)
    eg = o.grid(50, 50, 0.0, 0.0, 1.2, -9999.0)
    em = disc_mask(eg)
    with mk.Context(0) as ctx:
        ref, _, _ = run(ctx, x, y, w, hgrid, eg, em)
        peak = ctx.bytes_in_use
    fits = 0
    for budget in np.linspace(0.3 * peak, peak, 15).astype(np.int64):
        with mk.Context(0, hbm_budget=int(budget)) as ctx:
            try:
                got, _, _ = run(ctx, x, y, w, hgrid, eg, em)
            except mk.MgkError as e:
                assert e.status == -3
                continue
            fits += 1
            assert np.all(np.abs(got - ref) <= 1e-6 * np.abs(ref) + 1e-6)
    assert fits >= 2

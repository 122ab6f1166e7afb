"""The pass over the mask and the distance search at the sizes where they can
go wrong: widths around a ballot (32) and a trip (128), one row, one column,
NaN NoData; point and boundary counts on both sides of the all-pairs limit
(2^26), points outside the raster, distances limited to a reach.  Bit for bit
against the oracle (flags, distances; edge weights by their tests)."""
import numpy as np
import pytest

import oracle_py as o

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


def raster(ncols, nrows, kind, nodata=-9999.0, cs=2.0):
    g = o.grid(ncols, nrows, 10.0, 20.0, cs, nodata)
    r = np.random.default_rng(ncols * 1000 + nrows)
    m = np.ones((nrows, ncols), np.float32)
    if kind == "holes":
        m[r.random(m.shape) < 0.2] = nodata
    elif kind == "blocks":
        m[nrows // 3:nrows // 2, ncols // 4:ncols // 2] = nodata
    elif kind == "none":
        m[:] = nodata
    return g, m


@pytest.mark.parametrize("kind", ["full", "holes", "blocks", "none"])
@pytest.mark.parametrize("ncols,nrows", [(1, 1), (1, 40), (40, 1), (31, 7), (32, 8), (33, 9), (127, 33), (128, 5),
                                         (129, 66), (161, 3), (300, 130)])
def test_boundary_and_distances(ncols, nrows, kind):
    g, m = raster(ncols, nrows, kind)
    b = o.mark_boundary(g, m)
    r = np.random.default_rng(1)
    x = r.uniform(-10, 30 + 2 * ncols, 300).astype(np.float32)
    y = r.uniform(0, 40 + 2 * nrows, 300).astype(np.float32)
    with mk.Context(0) as ctx:
        ras = mk.Raster.upload(ctx, mk.Grid.of(g), m)
        for _ in range(2):  # marking again gives the same
            assert mk.mark_boundary(ctx, ras) == int(b.sum())
            assert np.array_equal(ras.boundary(), b)
        pts = mk.Points.upload(ctx, x, y)
        mk.calc_dist2_boundary(ctx, pts, ras)
        assert np.array_equal(pts.download(dist2=True, ew=False)[0], o.dist2_boundary(x, y, g, b))


@pytest.mark.parametrize("reach", [None, 25.0])
@pytest.mark.parametrize("n", [20_000, 90_000])
def test_distances_both_searches(n, reach):
    """About 2,400 boundary cells: 4.8e7 pairs are tried, 2.2e8 go through the lists."""
    g, m = raster(300, 300, "blocks")
    m[::9, ::7] = g.nodata
    b = o.mark_boundary(g, m)
    r = np.random.default_rng(n)
    x = r.uniform(-50, 700, n).astype(np.float32)
    y = r.uniform(-50, 700, n).astype(np.float32)
    ref = o.dist2_boundary(x, y, g, b)
    with mk.Context(0) as ctx:
        ras = mk.Raster.upload(ctx, mk.Grid.of(g), m)
        pts = mk.Points.upload(ctx, x, y)
        mk.calc_dist2_boundary(ctx, pts, ras, reach=reach)
        got = pts.download(dist2=True, ew=False)[0]
    if reach is None:
        assert np.array_equal(got, ref)
    else:
        near = ref <= reach * reach
        assert near.any() and not near.all()
        assert np.array_equal(got[near], ref[near]) and np.all(got[~near] > reach * reach)


def test_nan_nodata_marks_nothing_inside():
    g, m = raster(70, 50, "full", nodata=float("nan"))
    m[::3, ::5] = np.nan
    with mk.Context(0) as ctx:
        ras = mk.Raster.upload(ctx, mk.Grid.of(g), m)
        mk.mark_boundary(ctx, ras)
        assert np.array_equal(ras.boundary(), o.mark_boundary(g, m))

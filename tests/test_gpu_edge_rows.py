"""Edge weights where the row integral can go wrong: windows wider than one
prefix table (1,024 columns), rows of many valid runs, one-row and one-column
masks, and cell centres whose float rounding moves them by up to half a cell
(large coordinates), where the FP32 interval ends must yield to the exact
test.  Against the FP64 oracle: 1e-6 relative, the same points at exactly 1,
the same cell counts."""
import numpy as np
import pytest

import oracle_py as o

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


def mask_of(kind, g):
    m = np.ones((g.nrows, g.ncols), np.float32)
    r = np.random.default_rng(g.ncols + g.nrows)
    if kind == "holes":
        m[r.random(m.shape) < 0.3] = g.nodata
    elif kind == "stripes":  # up to ncols / 3 runs a row, the last column NoData
        m[:, ::3] = g.nodata
        m[::5] = 1.0
        m[:, -1] = g.nodata
    elif kind == "half":
        m[:, g.ncols // 2:] = g.nodata
    return m


@pytest.mark.parametrize("varh", [False, True])
@pytest.mark.parametrize("ncols,nrows,cs,org,h,kind", [
    (2600, 24, 1.0, 0.0, 500.0, "holes"),      # windows of three prefix tables
    (1025, 40, 1.0, 100.0, 200.0, "half"),
    (90, 70, 2.0, 0.0, 9.0, "stripes"),
    (300, 1, 1.0, 0.0, 12.0, "holes"),
    (1, 300, 1.0, 0.0, 12.0, "holes"),
    (64, 64, 0.25, 39_620.0, 1.7, "holes"),    # centres off by up to 1/128 cell
    (64, 64, 1.0, 500_000.0, 4.0, "half"),     # by 1/64 cell
    (64, 64, 1.0, 4_000_000.0, 5.0, "holes"),  # by 1/8 cell
    (64, 64, 0.3, 4_000_000.0, 1.5, "holes"),  # centres of neighbouring cells coincide
    (50, 50, 1.0, 0.0, 0.3, "holes"),          # less than a cell
])
def test_edge_weights_rows(ncols, nrows, cs, org, h, kind, varh):
    g = o.grid(ncols, nrows, org, org, cs, -9999.0)
    m = mask_of(kind, g)
    r = np.random.default_rng(7)
    n = 400
    x = (org + r.uniform(-2 * cs, (ncols + 2) * cs, n)).astype(np.float32)
    y = (org + r.uniform(-2 * cs, (nrows + 2) * cs, n)).astype(np.float32)
    # some points on cell centres and a whole number of cells plus 3h away from them
    x[:40] = (org + (r.integers(0, ncols, 40) + 0.5) * cs + 3.0 * np.float32(h)).astype(np.float32)
    y[:40] = (org + (r.integers(0, nrows, 40) + 0.5) * cs).astype(np.float32)
    hs = (h * r.uniform(0.5, 1.0, n)).astype(np.float32) if varh else None
    d2 = o.dist2_boundary(x, y, g, o.mark_boundary(g, m))
    ref, evals = o.edge_weights(x, y, h, d2, g, m, hs=hs)
    with mk.Context(0) as ctx:
        pts = mk.Points.upload(ctx, x, y, None, hs)
        ras = mk.Raster.upload(ctx, mk.Grid.of(g), m)
        mk.calc_dist2_boundary(ctx, pts, ras)
        count = mk.edge_correction_weights(ctx, pts, ras, 0.0 if varh else h, count=True)
        got = pts.download(ew=True)[1]
    assert count == evals
    fin = np.isfinite(ref)
    assert np.array_equal(np.isfinite(got), fin)
    assert np.array_equal(got == 1.0, ref.astype(np.float32) == 1.0)
    assert np.all(np.abs(got[fin] - ref[fin]) <= 1e-6 * np.abs(ref[fin]))

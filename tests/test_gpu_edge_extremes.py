"""Edge weights at bandwidths beyond the ordinary: NaN, and so large that the
squared reach leaves FP32.  NaN in, NaN out, for the points that have it alone;
where every cell lies deep inside the cutoff the factors are 1, and the weight
is 2 pi h^2 over the valid cells' area (1e-6, the parity tests' tolerance)."""
import numpy as np
import pytest

import oracle_py as o

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


def weights(x, y, g, m, h, hs=None):
    with mk.Context(0) as ctx:
        pts = mk.Points.upload(ctx, x, y, None, hs)
        ras = mk.Raster.upload(ctx, mk.Grid.of(g), m)
        mk.calc_dist2_boundary(ctx, pts, ras)
        mk.edge_correction_weights(ctx, pts, ras, h)
        return pts.download(ew=True)[1]


def study(n=200):
    g = o.grid(60, 45, 0.0, 0.0, 1.0, -9999.0)
    m = np.ones((45, 60), np.float32)
    m[:, 30:34] = g.nodata
    r = np.random.default_rng(n)
    return r.uniform(0, 60, n).astype(np.float32), r.uniform(0, 45, n).astype(np.float32), g, m


def test_nan_bandwidth_gives_nan_weights():
    x, y, g, m = study()
    assert np.isnan(weights(x, y, g, m, float("nan"))).all()
    hs = np.full(len(x), 3.0, np.float32)
    ref = weights(x, y, g, m, 0.0, hs)
    hs[::7] = np.nan
    got = weights(x, y, g, m, 0.0, hs)
    bad = np.isnan(hs)
    assert np.isnan(got[bad]).all() and np.array_equal(got[~bad], ref[~bad])


@pytest.mark.parametrize("varh", [False, True])
@pytest.mark.parametrize("h", [1e18, 6.0e18, 6.2e18, 9.0e18, 1.8e19])
def test_reach_beyond_fp32(h, varh):
    """9 h^2 is above FP32's range from h = 6.15e18, h^2 itself from 1.84e19."""
    x, y, g, m = study()
    got = weights(x, y, g, m, 0.0 if varh else h, np.full(len(x), h, np.float32) if varh else None)
    h2 = float(np.float32(h) * np.float32(h))
    ref = h2 * float(np.float32(6.283185307179586)) / (m == 1.0).sum()
    assert np.all(np.abs(got - ref) <= 1e-6 * ref)

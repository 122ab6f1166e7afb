"""Rasters in several tiles under budgets that hold the call's own buffers and
one tile's split blocks: the tiles that are planned first may take what a later
one needs, and give it back.  The raster is the unlimited one (1e-6 of each:
the parity tests' tolerance, twice)."""
import numpy as np
import pytest

import oracle_py as o

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu
NC, NR, H = 2311, 1873, 12.0


@pytest.fixture(scope="module")
def study():
    r = np.random.default_rng(1)
    c = r.uniform(0.15, 0.85, (12, 2)) * NR
    xy = c[r.integers(0, 12, 60_000)] + r.normal(0, 0.06 * NR, (60_000, 2))
    xy = np.clip(xy, 1.0, NR - 1.0).astype(np.float32)
    x, y, w = xy[:, 0].copy(), xy[:, 1].copy(), r.uniform(0.5, 2, 60_000).astype(np.float32)
    g = mk.Grid.of(o.grid(NC, NR, 0.0, 0.0, 1.0, -9999.0))
    with mk.Context(0) as ctx:
        return x, y, w, g, mk.kde_raster(ctx, x, y, w, H, g)[0]


@pytest.mark.parametrize("mib", [22, 26, 32, 40, 52, 64, 80])
def test_bands(study, mib):
    x, y, w, g, ref = study
    with mk.Context(0, hbm_budget=mib << 20) as ctx:
        got, _, _ = mk.kde_raster(ctx, x, y, w, H, g)
    assert np.all(np.abs(got - ref) <= 2e-6 * ref)


@pytest.mark.parametrize("mib", [10, 12, 16, 20, 24, 32])
@pytest.mark.parametrize("stream", [False, True])
def test_tiles(study, mib, stream):
    x, y, w, g, ref = study
    with mk.Context(0, hbm_budget=mib << 20) as ctx:
        if stream:
            got = np.empty((NR, NC), np.float32)
            pts = mk.Points.upload(ctx, x, y, w)
            mk.unit_edge_weights(ctx, pts)
            mk.density_stream(ctx, mk.Index(ctx, pts, H), g, 512, got)
        else:
            got, _, _ = mk.kde_raster(ctx, x, y, w, H, g, tile=512)
    assert np.all(np.abs(got - ref) <= 2e-6 * ref)

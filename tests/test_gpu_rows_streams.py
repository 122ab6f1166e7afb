"""A share of the rows whose inputs make the pool hand one block from stream to
stream: all the points' arrays are released while the rows' points are still
being gathered from them, and an edge mask of the same size class is then
copied in on the copy stream.  The rows are those of the whole raster (1e-6 of
each side: the parity tests' tolerance, twice)."""
import numpy as np
import pytest

import oracle_py as o

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [0, 128])
def test_rows_with_an_edge_mask_as_large_as_a_point_array(tile):
    n, side = 250_000, 500  # 1 MB each
    r = np.random.default_rng(2)
    x, y = r.uniform(0, 500, n).astype(np.float32), r.uniform(0, 500, n).astype(np.float32)
    w = r.uniform(0.5, 2.0, n).astype(np.float32)
    g = mk.Grid.of(o.grid(side, side, 0.0, 0.0, 1.0, -9999.0))
    em = np.ones((side, side), np.float32)
    em[200:210, 100:400] = -9999.0
    with mk.Context(0) as ctx:
        whole, _, _ = mk.kde_raster(ctx, x, y, w, 2.0, g, edge_grid=g, edge_mask=em, tile=tile)
        for _ in range(3):
            for row0, nr in ((0, 250), (250, 250), (100, 37)):
                part, _ = mk.kde_raster_rows(ctx, x, y, w, 2.0, g, row0, nr, edge_grid=g, edge_mask=em, tile=tile)
                ref = whole[row0:row0 + nr]
                assert np.all(np.abs(part - ref) <= 2e-6 * np.abs(ref))

"""Boundary distances where a raster's or a point's state is out of the
ordinary: points at infinity or NaN (no cell is nearest: DBL_MAX, on every
path), and a raster marked again after its mask has changed, with too little
memory for the new boundary (an error, then the right distances once there is
memory, never the old cells)."""
import numpy as np
import pytest

import oracle_py as o

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


# all pairs in one part, all pairs in several, the bins' lists
@pytest.mark.parametrize("n,side", [(12, 40), (12, 400), (200_000, 400)])
def test_points_without_a_nearest_cell(n, side):
    g = o.grid(side, side, 0.0, 0.0, 1.0, -9999.0)
    m = np.ones((side, side), np.float32)
    r = np.random.default_rng(n)
    x, y = r.uniform(0, side, n).astype(np.float32), r.uniform(0, side, n).astype(np.float32)
    ref = o.dist2_boundary(x, y, g, o.mark_boundary(g, m))
    bad = [(np.inf, 1.0), (1.0, -np.inf), (np.nan, 2.0), (3.0, np.nan), (np.inf, np.nan)]
    for i, (px, py) in enumerate(bad):
        x[2 * i], y[2 * i] = px, py
        ref[2 * i] = np.finfo(np.float64).max
    with mk.Context(0) as ctx:
        pts = mk.Points.upload(ctx, x, y)
        ras = mk.Raster.upload(ctx, mk.Grid.of(g), m)
        mk.calc_dist2_boundary(ctx, pts, ras)
        assert np.array_equal(pts.download(dist2=True, ew=False)[0], ref)


def test_marked_again_without_memory():
    side = 300
    g = o.grid(side, side, 0.0, 0.0, 1.0, -9999.0)
    r = np.random.default_rng(8)
    x, y = r.uniform(0, side, 5000).astype(np.float32), r.uniform(0, side, 5000).astype(np.float32)
    plain = np.ones((side, side), np.float32)  # a ring of 1,196 cells, 10 KB of them
    holes = np.where(r.random((side, side)) < 0.2, g.nodata, 1.0).astype(np.float32)  # most cells, 500 KB
    ref = o.dist2_boundary(x, y, g, o.mark_boundary(g, holes))
    refused = 0
    for kib in range(512, 4096, 128):
        mask = torch.from_numpy(plain).cuda()
        with mk.Context(0, hbm_budget=kib << 10) as ctx:
            try:
                pts = mk.Points.upload(ctx, x, y)
                ras = mk.Raster.wrap(ctx, mk.Grid.of(g), mask)
                mk.mark_boundary(ctx, ras)
            except mk.MgkError as e:
                assert e.status == -3
                continue
            mask.copy_(torch.from_numpy(holes))
            torch.cuda.synchronize()
            try:
                mk.mark_boundary(ctx, ras)
            except mk.MgkError as e:
                assert e.status == -3
                refused += 1
            try:
                mk.calc_dist2_boundary(ctx, pts, ras)
            except mk.MgkError as e:
                assert e.status == -3
                continue
            assert np.array_equal(pts.download(dist2=True, ew=False)[0], ref)
    assert refused >= 1


def test_marked_on_one_stream_read_on_another():
    side = 900
    g = o.grid(side, side, 0.0, 0.0, 1.0, -9999.0)
    r = np.random.default_rng(5)
    m = np.where(r.random((side, side)) < 0.1, g.nodata, 1.0).astype(np.float32)
    x, y = r.uniform(0, side, 100).astype(np.float32), r.uniform(0, side, 100).astype(np.float32)
    bm = o.mark_boundary(g, m)
    ref = o.dist2_boundary(x, y, g, bm)
    ew, _ = o.edge_weights(x, y, 9.0, ref, g, m)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with mk.Context(0, stream=a) as ctx:
        pts = mk.Points.upload(ctx, x, y)
        ras = mk.Raster.upload(ctx, mk.Grid.of(g), m)
        assert mk.mark_boundary(ctx, ras) == int(np.count_nonzero(bm))
        ctx.set_stream(b)
        mk.calc_dist2_boundary(ctx, pts, ras)
        mk.edge_correction_weights(ctx, pts, ras, 9.0)
        d2, got = pts.download(dist2=True)
    assert np.array_equal(d2, ref)
    assert np.all(np.abs(got - ew) <= 1e-6 * np.abs(ew))

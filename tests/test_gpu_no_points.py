"""Calls without a single point: the likelihoods of a batch and of a share are
empty sums, the golden section closes on its bracket, densities are zero."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edge", [False, True])
def test_no_points(edge):
    none = np.zeros(0, np.float32)
    g = mk.Grid(70, 50, 0.0, 0.0, 1.0, -9999.0)
    m = np.ones((50, 70), np.float32)
    with mk.Context(0) as ctx:
        pts, ras = mk.Points.upload(ctx, none, none), None
        if edge:
            ras = mk.Raster.upload(ctx, g, m)
            mk.calc_dist2_boundary(ctx, pts, ras)
            assert mk.edge_correction_weights(ctx, pts, ras, 3.0, count=True) == 0
        for hs in ([1.0], [1.0, 2.0, 4.0]):
            logl, best = mk.log_likelihood_batch(ctx, pts, ras, hs)
            assert np.all(logl == 0.0) and best == 0 and ctx.last_loo_evals == (0, 0)
        h, iterations = mk.mle_fixed_bandwidth(ctx, pts, ras, 3.0)
        assert 0.15 < h < 6.0 and iterations > 5
        d_ew = torch.zeros(64, device="cuda")
        torch.cuda.synchronize()
        part, ev = mk.loo_share_loglik(ctx, pts, [1.0, 2.0], 1, 2, d_ew if edge else None)
        assert np.all(part == 0.0) and ev == 0
        den, _, ev = mk.kde_raster(ctx, none, none, None, 3.0, g, m, g if edge else None, m if edge else None, count=True)
        assert np.all(den == 0.0) and ev == 0

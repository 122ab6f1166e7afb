"""Small tiles split batch by batch (64 candidates) or two by two: blocks of one
to five batches, one block and several, per-point bandwidths, and a batch of
tiles against single ones.  Against the FP64 oracle (1e-6 relative, the parity
tests' tolerance), pair counts equal."""
import numpy as np
import pytest

import oracle_py as o

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("varh", [False, True])
@pytest.mark.parametrize("n,ncols,nrows", [(64, 100, 60), (128, 100, 60), (129, 100, 60), (320, 128, 64), (700, 260, 130),
                                           (3000, 500, 400), (9000, 700, 600), (20_000, 700, 600)])
def test_small_tiles(n, ncols, nrows, varh):
    r = np.random.default_rng(n)
    x, y = r.uniform(0, ncols, n).astype(np.float32), r.uniform(0, nrows, n).astype(np.float32)
    w = r.lognormal(0, 0.5, n).astype(np.float32)
    h = 7.0
    hs = (h * r.uniform(0.5, 1.5, n)).astype(np.float32) if varh else None
    g = o.grid(ncols, nrows, 0.0, 0.0, 1.0, -9999.0)
    ref, evals = o.density(x, y, w, np.ones(n), h, g, hs=hs) if varh else o.density(x, y, w, np.ones(n), h, g)
    with mk.Context(0) as ctx:
        pts = mk.Points.upload(ctx, x, y, w, hs)
        mk.unit_edge_weights(ctx, pts)
        idx = mk.Index(ctx, pts, 0.0 if varh else h)
        out, two = torch.empty(nrows, ncols, device="cuda"), [torch.empty(nrows, ncols, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        assert mk.density_tile(ctx, idx, mk.Grid.of(g), 0, 0, nrows, ncols, None, out, count=True) == evals
        mk.density_tiles(ctx, [(idx, mk.Grid.of(g), 0, 0, nrows, ncols, None, t) for t in two])
        got = out.cpu().numpy().astype(np.float64)
        for t in two:
            assert torch.equal(t, out)
    assert np.array_equal(got == 0, ref == 0)
    assert (np.abs(got - ref) / np.maximum(ref, 1e-300)).max() <= 1e-6

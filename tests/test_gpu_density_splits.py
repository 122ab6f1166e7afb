"""How a tile's blocks are split into work items: blocks of candidates around
the smallest (256) and the largest (2,048) least split size, single tiles and
batches, and budgets too small for the finer split.  Against the FP64 oracle
(1e-6 relative, the parity tests' tolerance), pair counts equal."""
import numpy as np
import pytest

import oracle_py as o

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu
H = 6.0


def points(n):
    """Most of the points in one block, a few spread."""
    r = np.random.default_rng(n)
    k = n - n // 10
    x = np.concatenate([r.uniform(20, 100, k), r.uniform(0, 300, n - k)])
    y = np.concatenate([r.uniform(100, 130, k), r.uniform(0, 200, n - k)])
    return x.astype(np.float32), y.astype(np.float32), r.lognormal(0, 0.5, n).astype(np.float32)


def check(got, ref):
    assert np.array_equal(got == 0, ref == 0)
    assert (np.abs(got - ref) / np.maximum(ref, 1e-300)).max() <= 1e-6


@pytest.mark.parametrize("n", [63, 255, 257, 300, 513, 2047, 2300, 9000, 200_000])
def test_split_sizes(n):
    x, y, w = points(n)
    g = o.grid(300, 200, 0.0, 0.0, 1.0, -9999.0)
    ref, evals = o.density(x, y, w, np.ones(n), H, g)
    with mk.Context(0) as ctx:
        pts = mk.Points.upload(ctx, x, y, w)
        mk.unit_edge_weights(ctx, pts)
        idx = mk.Index(ctx, pts, H)
        out = torch.empty(200, 300, device="cuda")
        two = [torch.empty(200, 300, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        assert mk.density_tile(ctx, idx, mk.Grid.of(g), 0, 0, 200, 300, None, out, count=True) == evals
        mk.density_tiles(ctx, [(idx, mk.Grid.of(g), 0, 0, 200, 300, None, t) for t in two])
        check(out.cpu().numpy().astype(np.float64), ref)
        for t in two:  # a tile is planned the same alone and in a batch
            assert torch.equal(t, out)


def test_split_under_small_budgets():
    """At every budget the call either says so or gives the right raster."""
    x, y, w = points(20_000)
    g = o.grid(300, 200, 0.0, 0.0, 1.0, -9999.0)
    ref, _ = o.density(x, y, w, np.ones(len(x)), H, g)
    fits = 0
    for mib in (3, 6, 8, 10, 12, 16, 24, 48, 96):
        with mk.Context(0, hbm_budget=mib << 20) as ctx:
            try:
                den, _, _ = mk.kde_raster(ctx, x, y, w, H, mk.Grid.of(g), tile=300)
            except mk.MgkError as e:
                assert e.status == -3
                continue
            fits += 1
            check(den.astype(np.float64), ref)
    assert fits >= 3

"""A batch of tiles under budgets too small for all its split blocks at once:
each tile as it is alone, bit for bit, and no batch refused whose tiles are
accepted one by one."""
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


def test_batch_is_each_tile_alone_at_every_budget():
    x, y, w = points(9000)
    rows = [(0, 200), (64, 136), (0, 130), (30, 100), (0, 64)]
    g = mk.Grid.of(o.grid(300, 200, 0.0, 0.0, 1.0, -9999.0))
    plain, split = [], 0
    for kib in [1 << 20, *range(1024, 14 << 10, 512), *range(14 << 10, 128 << 10, 3 << 10)]:
        with mk.Context(0, hbm_budget=(kib << 10) + 100_000) as ctx:
            try:
                pts = mk.Points.upload(ctx, x, y, w)
                mk.unit_edge_weights(ctx, pts)
                idx = mk.Index(ctx, pts, H)
                alone = [torch.empty(nr, 300, device="cuda") for _, nr in rows]
                ev = [mk.density_tile(ctx, idx, g, r0, 0, nr, 300, None, t, count=True)
                      for (r0, nr), t in zip(rows, alone)]
            except mk.MgkError as e:
                assert e.status == -3
                continue
            batch = [torch.empty(nr, 300, device="cuda") for _, nr in rows]
            torch.cuda.synchronize()
            assert ev == mk.density_tiles(ctx, [(idx, g, r0, 0, nr, 300, None, t) for (r0, nr), t in zip(rows, batch)],
                                          count=True)
            for a, b in zip(alone, batch):
                assert torch.equal(a, b)
            plain = plain or alone
            split += all(torch.equal(a, b) for a, b in zip(alone, plain))
    assert split >= 3  # budgets at which the tiles keep the plans of an unlimited one

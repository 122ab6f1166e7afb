"""The levels of a bandwidth batch built together (fewer than 2^19 points) and
one after the other, at counts around a sort tile of 256, 1,024 and 4,096
items and on both sides of the line: the pairs that each batch scans have to
be all pairs within 3h, and every h of a batch over several octaves has to get
what it gets alone, on a single level.  The scan's partial sums are FP32 over
at most 128 candidates (2^-17 of a sum of one sign), FP64 above: the mean log
agrees within 2 x 2^-17."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h0,octaves", [(2, 3.0, 8), (255, 40.0, 3), (257, 9.0, 5), (4097, 2.0, 7), (65_535, 0.5, 5),
                                          (65_537, 0.6, 4), (524_287, 0.2, 3), (524_288, 0.2, 3)])
def test_levels_hold_every_point_once(n, h0, octaves):
    r = np.random.default_rng(n)
    x, y = r.uniform(0, 1000, n), r.uniform(0, 700, n)
    x[: n // 3], y[: n // 3] = 400.0 + 20 * r.standard_normal(n // 3), 300.0 + 20 * r.standard_normal(n // 3)
    if n > 100_000:  # spread out: the coarsest level's pairs stay few
        x, y = r.uniform(0, 1000, n), r.uniform(0, 700, n)
    x, y, w = (torch.from_numpy(a.astype(np.float32)).cuda() for a in (x, y, r.lognormal(0, 0.5, n)))
    hs = [h0 * 2.0 ** k for k in range(octaves)]
    torch.cuda.synchronize()
    with mk.Context(0) as ctx:
        pts = mk.Points.wrap(ctx, x, y, w)
        got, _ = mk.log_likelihood_batch(ctx, pts, None, hs)
        pairs = ctx.last_loo_evals[1]
        alone, count = [], 0
        for h in hs:
            alone.append(mk.log_likelihood_batch(ctx, pts, None, [h])[0][0])
            count += ctx.last_loo_evals[1]
    assert pairs == count
    if n <= 65_537:
        ref = 0
        for p in range(0, n, 2048):
            d2 = (x[p:p + 2048, None].double() - x.double()) ** 2 + (y[p:p + 2048, None].double() - y.double()) ** 2
            ref += sum(int((d2 < 9.0 * float(np.float32(h) * np.float32(h))).sum()) for h in hs)
        assert pairs == ref - n * octaves
    assert np.abs(np.asarray(got) - np.asarray(alone)).max() <= 2 * 2.0 ** -17 * n

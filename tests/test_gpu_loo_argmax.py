"""The last step of a bandwidth batch: one to several warps of bandwidths, ties
(the first index of the largest), and the counts and values of a second run
after a first with other bandwidths."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 40, 3000])
@pytest.mark.parametrize("nh", [1, 2, 31, 33, 100])
def test_argmax_takes_the_first_of_the_largest(n, nh):
    r = np.random.default_rng(nh)
    x, y = (torch.from_numpy(r.uniform(0, 100, n).astype(np.float32)).cuda() for _ in range(2))
    hs = np.float32(2.0) * np.float32(1.15) ** r.integers(0, 12, nh).astype(np.float32)  # most of them twice and more
    torch.cuda.synchronize()
    with mk.Context(0) as ctx:
        pts = mk.Points.wrap(ctx, x, y, None)
        first, best = mk.log_likelihood_batch(ctx, pts, None, hs)
        evals = tuple(ctx.last_loo_evals)
        assert best == int(np.argmax(first))
        mk.log_likelihood_batch(ctx, pts, None, hs[::-1] * np.float32(1.5))
        again, b2 = mk.log_likelihood_batch(ctx, pts, None, hs)
        assert b2 == best and np.array_equal(first, again) and tuple(ctx.last_loo_evals) == evals

"""The pieces in which the adaptive likelihood's point densities are summed in
plain FP32 before each compensated step: at most 32 candidates."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import mgpukde_tiled_b200 as mk  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heavy", [0, 32])
def test_pieces_of_at_most_32(heavy):
    """65 points in one place, one of them 2^25 times as heavy as the others.
    An FP32 sum that holds it loses each light term added to it, 2^-25 of the
    sum, up to the end of the piece: 31 at most.  The bandwidths are all h to a
    rounding (2^-23 in h^2), the terms' weights rounded once (the light ones by
    the same factor as the heavy one, a power of two apart)."""
    n, h = 65, 3.0
    w = np.ones(n, np.float32)
    w[heavy] = 2.0 ** 25
    x, y = np.full(n, 17.0, np.float32), np.full(n, 5.0, np.float32)
    with mk.Context(0) as ctx:
        got = mk.loglik_adaptive(ctx, mk.Points.upload(ctx, x, y, w), None, h, -0.5)
    two_pi = float(np.float32(6.283185307179586))
    ref = np.log((w.sum(dtype=np.float64) - w.astype(np.float64)) / (h * h * two_pi)).sum()
    assert abs(got - ref) <= n * (31 * 2.0 ** -25 + 2 * 2.0 ** -23)

"""GPU tests of clear_inner_layer's grouped search (csrc/clear_inner.cu) at the edges of its 32-panel groups, with the
panels out of order, and where more panels tie than its list holds, bit for bit against the oracle."""
import numpy as np
import pytest

import omega2d_gb300 as og

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npan", [3, 31, 32, 33, 64, 65, 1025, 1057])
@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("n", [1, 77, 6001])
def test_clear_groups_match_oracle(ctx, restatement, npan, shuffled, n):
    rng = np.random.default_rng(npan + n)
    body = og.circle_panels(npan)
    if shuffled:
        body.idx = body.idx.reshape(-1, 2)[rng.permutation(npan)].ravel().copy()
    rad, a = rng.uniform(0.3, 1.5, n), rng.uniform(0, 2 * np.pi, n)
    x, y = (rad * np.cos(a)).astype(np.float32), (rad * np.sin(a)).astype(np.float32)
    if n > 1:
        x[0] = y[0] = 0.0                    # the centre: every panel within rounding of the closest
        x[1], y[1] = body.nx[0], body.ny[0]  # on a node
    s = rng.normal(0, 1, n).astype(np.float32)
    r = np.full(n, 0.01, np.float32)
    for method in (0, 1):
        p = og.Points(x, y, r, s)
        lost, nc = og.clear_inner_layer(p, body, 0.01, method=method, env=og.ExecEnv(context=ctx))
        ox, oy, os_, olost, onc = restatement.clear_inner(method, og.CLEAR_CUTOFF, 0.01, body.nx, body.ny, body.idx,
                                                          x, y, s, r)
        np.testing.assert_array_equal(p.x, ox)
        np.testing.assert_array_equal(p.y, oy)
        np.testing.assert_array_equal(p.s, os_)
        assert nc == onc
        assert abs(lost - olost) < 1e-4 * max(1.0, abs(olost))

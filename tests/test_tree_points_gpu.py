"""GPU tests of the treecode's nodes of radius 0 (csrc/tree.cu): a last leaf with one source, and leaves of coincident
sources, under parents whose radius is small, so that its inverse powers leave FP32's range."""
import numpy as np
import pytest

import omega2d_gb300 as og
from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 2e-6          # the treecode's tolerance in tests/test_tree_gpu.py: truncation 1.2e-7 and FP32 pairs


# n % 32 == 1: one source in the last leaf; coincident: the first of them at one point (two whole leaves)
@pytest.mark.parametrize("n,unit,coincident", [(500_033, 1.0, 0), (1_000_001, 1.0, 0), (20_001, 1e-3, 0), (60_001, 1e-3, 0),
                                               (100_000, 1.0, 96), (100_000, 1e-3, 96)])
def test_nodes_of_radius_zero(ctx, n, unit, coincident):
    rng = np.random.default_rng(n)
    x, y = (unit * rng.uniform(-1, 1, (2, n))).astype(np.float32)
    x[:coincident], y[:coincident] = x[:1], y[:1]
    r = np.full(n, 0.004 * unit, np.float32)
    s = rng.normal(0, 1 / np.sqrt(n), n).astype(np.float32)
    env = og.ExecEnv(og.CORE_GAUSSIAN, og.COMPENSATED, ctx)
    a, b = og.Points(x, y, r, s), og.Points(x, y, r, s)
    og.points_affect_points_tree(a, a, env)
    og.points_affect_points(b, b, og.VELONLY, env)
    assert np.isfinite(a.u).all() and np.isfinite(a.v).all()
    assert rel_err(b.u, a.u) < TOL and rel_err(b.v, a.v) < TOL

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


@pytest.mark.parametrize("order", [2, 4, 6, 12])
def test_distant_nodes_keep_their_terms(ctx, order):
    """A leaf of radius 0.1 with its strength at one end, 0.35 from the targets: P terms leave at most |w|^P / (1 - |w|)
    of sum |G| / |d|, |w| = 0.1 / 0.35, whatever theta is."""
    sx = np.concatenate([[-0.1], np.full(31, 0.1)]).astype(np.float32)
    sy, r = np.zeros(32, np.float32), np.full(32, 1e-3, np.float32)
    s = np.concatenate([[1e-3], np.full(31, 1.0)]).astype(np.float32)
    t = og.Points(np.linspace(0.35, 0.3501, 64).astype(np.float32), np.zeros(64, np.float32), np.full(64, 1e-3, np.float32))
    og.points_affect_points_tree(og.Points(sx, sy, r, s), t, og.ExecEnv(og.CORE_GAUSSIAN, og.COMPENSATED, ctx), theta=0.7,
                                 order=order)
    d = t.x.astype(np.float64)[:, None] - sx.astype(np.float64)[None, :]
    terms, w = s / np.abs(d), 0.1 / 0.35
    err = np.abs(t.v - (s / d).sum(1))
    assert np.all(err <= (w ** order / (1 - w) + 2e-6) * terms.sum(1))     # 2e-6: FP32, as TOL


def test_node_strengths_cancel(ctx):
    """Four leaves at one point whose strengths add up to 2^24, 1, -2^24 and 0: their node has strength 1."""
    s = np.concatenate([np.full(32, 2.0 ** 19), [1.0], np.zeros(31), np.full(32, -2.0 ** 19), np.zeros(32)]).astype(np.float32)
    z, r = np.zeros(128, np.float32), np.full(128, 1e-3, np.float32)
    d = np.linspace(1.0, 1.001, 64).astype(np.float32)
    t = og.Points(d, np.zeros(64, np.float32), np.full(64, 1e-3, np.float32))
    og.points_affect_points_tree(og.Points(z, z, r, s), t, og.ExecEnv(og.CORE_GAUSSIAN, og.COMPENSATED, ctx))
    assert np.all(np.abs(t.v * d - 1.0) < 2e-6) and np.all(np.abs(t.u) < 2e-6)

"""GPU tests of the treecode's target groups (csrc/tree.cu: 64 targets per warp, one, two or four warps per group) at
their edges, against the FP64 oracle and the direct sum."""
import numpy as np
import pytest

import omega2d_gb300 as og
from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 2e-6          # the treecode's tolerance in tests/test_tree_gpu.py: truncation 1.2e-7 and FP32 pairs


def vortices(n, seed, rad=0.02):
    rng = np.random.default_rng(seed)
    x, y = rng.uniform(-1, 1, (2, n)).astype(np.float32)
    return x, y, np.full(n, rad, np.float32), rng.normal(0, 1 / np.sqrt(n), n).astype(np.float32)


@pytest.mark.parametrize("core", [og.CORE_GAUSSIAN, og.CORE_V2, og.CORE_SINGULAR])
@pytest.mark.parametrize("ns,nt", [(1, 1), (31, 63), (33, 65), (2049, 64), (5000, 129), (127, 1000)])
@pytest.mark.parametrize("thick", [True, False])
def test_tree_group_edges(ctx, restatement, core, ns, nt, thick):
    x, y, r, s = vortices(ns, ns + nt)
    tx, ty, tr, _ = vortices(nt, 7 * nt)
    t = og.Points(tx, ty, tr if thick else None)
    og.points_affect_points_tree(og.Points(x, y, r, s), t, og.ExecEnv(core, context=ctx))
    u, v, _ = restatement.points_affect_points(core, 1, x, y, r, s, tx, ty, tr if thick else None, fp64=True)
    assert rel_err(u, t.u) < TOL and rel_err(v, t.v) < TOL


@pytest.mark.parametrize("n", [40_001, 80_003, 160_001])      # four, two and one warp per group
def test_tree_matches_direct(ctx, n):
    x, y, r, s = vortices(n, n, 0.004)
    env = og.ExecEnv(og.CORE_GAUSSIAN, og.COMPENSATED, ctx)
    a, b = og.Points(x, y, r, s), og.Points(x, y, r, s)
    og.points_affect_points_tree(a, a, env)
    og.points_affect_points(b, b, og.VELONLY, env)
    assert rel_err(b.u, a.u) < TOL and rel_err(b.v, a.v) < TOL


@pytest.mark.parametrize("x", [0.0, 0.0009, 0.00095, 0.00103, 0.0011, 0.01])
def test_tree_leaves_about_the_core(ctx, restatement, x):
    # a leaf at d^2 / s^2 = x from the targets: below 0.001 the Gaussian core is the constant 1 / s^2, which is 4.7e-4
    # off (1 - e^-x) / d^2 there; that formula in FP32 carries 2^-23 / x <= 1.2e-4 (the FP64 oracle none)
    rad = np.float32(0.02)
    d = np.float32(np.sqrt(2 * x) * rad)
    sx = np.concatenate([np.full(32, d), np.full(32, 0.3)]).astype(np.float32)
    sy, r, s = np.zeros(64, np.float32), np.full(64, rad), np.full(64, 1 / 64, np.float32)
    t = og.Points(np.zeros(64, np.float32), np.full(64, 1e-7, np.float32), r)
    og.points_affect_points_tree(og.Points(sx, sy, r, s), t, og.ExecEnv(og.CORE_GAUSSIAN, context=ctx))
    u, v, _ = restatement.points_affect_points(og.CORE_GAUSSIAN, 1, sx, sy, r, s, t.x, t.y, r, fp64=True)
    assert np.isfinite(t.u).all() and rel_err(v, t.v) < 2e-4

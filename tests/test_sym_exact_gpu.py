"""GPU tests of the precision of the compensated pair-once sums (csrc/p2p_sym.cuh, sym_moments.cuh): two clusters of
coincident particles whose pairs evaluate without rounding (d^2 and K are powers of two) and whose strengths are whole
numbers.  A row's sum over 32 columns and a column's over half a warp's rows stay below 2^24; a row block's sums reach
2^26 and cancel between the blocks.  Kept in two-sums they cancel exactly; one FP32 number per row block is some units
off a total of about 1e6."""
import numpy as np
import pytest

import omega2d_gb300 as og

pytestmark = pytest.mark.gpu


def clusters(n, block, top, seed):
    """n - block particles at (0, 0), strengths of one sign per row block, then a block of them at (0.5, 0.5)."""
    rng = np.random.default_rng(seed)
    x = np.where(np.arange(n) < n - block, 0.0, 0.5).astype(np.float32)
    g = rng.integers(top // 4, top // 2, n) * 2.0 + 1.0
    g *= np.where(np.arange(n) // block % 2, -1.0, 1.0)
    total = g[:n - block].sum()
    assert abs(total) < 2 ** 24 and g.astype(np.float32).astype(np.float64).tolist() == g.tolist()
    return x, x.copy(), g, total


# 1024 and 2048 rows a block (four and eight row pairs a thread): half a warp's rows are 128 and 256 of them
@pytest.mark.parametrize("n,block,top", [(9 * 1024, 1024, 2 ** 17), (17 * 2048, 2048, 2 ** 16)])
@pytest.mark.parametrize("seed", [1, 2])
def test_velocity_columns_are_exact(ctx, n, block, top, seed):
    x, y, g, total = clusters(n, block, top, seed)
    p = og.Points(x, y, np.full(n, 1e-3, np.float32), g.astype(np.float32))
    og.points_affect_points(p, p, og.VELONLY, og.ExecEnv(og.CORE_SINGULAR, og.COMPENSATED, ctx))
    # K = 2, K d = (1, 1): u = -sum G, v = sum G
    assert np.all(p.u[n - block:] == -total) and np.all(p.v[n - block:] == total)


@pytest.mark.parametrize("seed", [1, 2])
def test_gradient_columns_are_exact(ctx, seed):
    n, block = 19 * 512, 512
    x, y, g, total = clusters(n, block, 2 ** 17, seed)
    p = og.Points(x, y, np.full(n, 1e-3, np.float32), g.astype(np.float32))
    og.points_affect_points(p, p, og.VELANDGRAD, og.ExecEnv(og.CORE_GAUSSIAN, og.COMPENSATED, ctx))
    assert np.all(p.u[n - block:] == -total) and np.all(p.v[n - block:] == total)
    # du/dx = 2 K^2 dx dy sum G = -dv/dy; the coincident pairs add nothing to these two
    assert np.all(p.grad[0][n - block:] == 2.0 * total) and np.all(p.grad[3][n - block:] == -2.0 * total)


@pytest.mark.parametrize("seed", [1, 2])
def test_vjp_columns_are_exact(ctx, seed):
    n, block = 21 * 512, 512
    x, y, g, total = clusters(n, block, 2 ** 16, seed)
    g[n - block:] = 0.0
    p = og.Points(x, y, np.full(n, 1e-3, np.float32), g.astype(np.float32))
    lu, lv = np.full(n, -1.0, np.float32), np.ones(n, np.float32)
    gx, gy, _ = og.points_affect_points_vjp_self(p, lu, lv, og.ExecEnv(og.CORE_GAUSSIAN, og.COMPENSATED, ctx))
    # v - u = sum G (dx + dy) / d^2 / (2 pi): its derivative by x is sum G (1/d^2 - 2 dx (dx + dy) / d^4) / (2 pi)
    want = -2.0 * total / (2.0 * np.pi)
    for got in (gx, gy):
        assert np.all(np.abs(got[n - block:] - want) <= 2.0 ** -23 * abs(want))     # one FP32 rounding of the result


@pytest.mark.parametrize("accum", [og.COMPENSATED, og.PLAIN_F32])
def test_vjp_of_a_particle_with_itself_is_none(ctx, restatement, accum):
    """Particles a million radii apart: the core at distance 0 is 1e14 times as large as between them, so anything left
    of a particle's weight with itself would be all there is."""
    n = 12_001
    rng = np.random.default_rng(n)
    x, y = (1e6 * rng.uniform(-1, 1, (2, n))).astype(np.float32)
    r, s = np.full(n, 0.02, np.float32), rng.normal(0, 1, n).astype(np.float32)
    lu, lv = rng.normal(0, 1, (2, n)).astype(np.float32)
    got = og.points_affect_points_vjp_self(og.Points(x, y, r, s), lu, lv, og.ExecEnv(og.CORE_GAUSSIAN, accum, ctx))
    for a, b in zip(restatement.self_vjp(og.CORE_GAUSSIAN, x, y, r, s, lu, lv), got):
        assert np.max(np.abs(a - b)) < (2e-5 if accum == og.COMPENSATED else 1e-4) * np.max(np.abs(a))   # as test_sym_gpu.py

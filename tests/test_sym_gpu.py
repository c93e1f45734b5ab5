"""GPU tests of the self-interaction sums that evaluate each unordered pair once (csrc/p2p_sym.cuh, sym_moments.cuh), at
the edges of their 32-column groups and 1024- or 512-row blocks and over several passes, against the FP64 oracle and the
one-sided kernels."""
import numpy as np
import pytest

import omega2d_gb300 as og
from conftest import rel_err

pytestmark = pytest.mark.gpu

CORES = [og.CORE_RM, og.CORE_GAUSSIAN, og.CORE_V2, og.CORE_WL, og.CORE_V3, og.CORE_SINGULAR, og.CORE_COMPACT_EXP]


def cloud(n, seed, spread, rad=0.02):
    rng = np.random.default_rng(seed)
    x, y = rng.uniform(-1, 1, (2, n)).astype(np.float32)
    r = (rad * rng.uniform(1 - spread, 1 + spread, n)).astype(np.float32)
    return x, y, r, rng.normal(0, 1 / np.sqrt(n), n).astype(np.float32)


def self_velocity(ctx, core, accum, x, y, r, s):
    p = og.Points(x, y, r, s, u=np.full(x.size, 0.5, np.float32))
    og.points_affect_points(p, p, og.VELONLY, og.ExecEnv(core, accum, ctx), finalize=True, fs=(1.0, -0.25))
    return p.u, p.v


# the tolerances of the packed kernels' tests: FP32 pairs with compensated or plain sums
@pytest.mark.parametrize("core", CORES)
@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 2e-6), (og.PLAIN_F32, 2e-5)])
@pytest.mark.parametrize("n,spread", [(1, 0.0), (2, 0.5), (33, 0.0), (1023, 0.5), (1025, 0.0), (2081, 0.5), (5121, 0.0)])
def test_self_sum_matches_fp64(ctx, restatement, core, accum, tol, n, spread):
    x, y, r, s = cloud(n, 7 * n + core, spread)
    if n > 1024:                       # coincident particles, in one block and in two
        x[5], y[5] = x[0], y[0]
        x[n - 1], y[n - 1] = x[1], y[1]
    u, v = self_velocity(ctx, core, accum, x, y, r, s)
    u64, v64, _ = restatement.points_affect_points(core, 1, x, y, r, s, x, y, r, fp64=True, tu=np.full(n, 0.5),
                                                   tv=np.zeros(n))
    assert rel_err(1.0 + u64 / (2 * np.pi), u) < tol
    assert rel_err(-0.25 + v64 / (2 * np.pi), v) < tol


@pytest.mark.parametrize("core,n,spread", [(og.CORE_GAUSSIAN, 400_003, 0.0), (og.CORE_V2, 390_001, 0.5)])
def test_several_passes_match_one_sided(ctx, core, n, spread):
    """More row blocks than one pass holds: the running sums carry over, and a repeat gives the same bits."""
    x, y, r, s = cloud(n, n, spread, 0.004)
    u, v = self_velocity(ctx, core, og.COMPENSATED, x, y, r, s)
    u2, v2 = self_velocity(ctx, core, og.COMPENSATED, x, y, r, s)
    assert np.array_equal(u, u2) and np.array_equal(v, v2)
    try:
        ctx.set_kernel_variant(og.VARIANT_PACKED4)
        uo, vo = self_velocity(ctx, core, og.COMPENSATED, x, y, r, s)
    finally:
        ctx.set_kernel_variant(og.VARIANT_AUTO)
    assert rel_err(uo, u) < 2e-6 and rel_err(vo, v) < 2e-6


# sizes past the one-launch kernels: one row over a block, an odd remainder
@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 2e-6), (og.PLAIN_F32, 2e-5)])
@pytest.mark.parametrize("res", [og.VELANDGRAD, og.VELANDVORT, og.VELANDSHEAR])
@pytest.mark.parametrize("n,spread", [(9217, 0.0), (9999, 0.5), (18_001, 0.0)])
def test_self_results_match_generic(ctx, accum, tol, res, n, spread):
    x, y, r, s = cloud(n, n + res, spread)
    x[n - 1], y[n - 1] = x[1], y[1]    # coincident particles
    outs = []
    try:
        for variant in (og.VARIANT_GENERIC, og.VARIANT_AUTO):
            ctx.set_kernel_variant(variant)
            p = og.Points(x, y, r, s)
            og.points_affect_points(p, p, res, og.ExecEnv(og.CORE_GAUSSIAN, accum, ctx), finalize=True, fs=(1.0, -0.25))
            outs.append([p.u, p.v] + [a for a in (p.vort, p.shear) if a is not None] + list(p.grad or []))
    finally:
        ctx.set_kernel_variant(og.VARIANT_AUTO)
    for a, b in zip(*outs):
        assert rel_err(a, b) < tol


@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 2e-5), (og.PLAIN_F32, 1e-4)])    # as tests/test_adjoint_packed_gpu.py
@pytest.mark.parametrize("n,spread", [(10_241, 0.0), (12_001, 0.5), (18_001, 0.0)])
def test_self_vjp_matches_fp64(ctx, restatement, accum, tol, n, spread):
    x, y, r, s = cloud(n, n, spread)
    lu, lv = np.random.default_rng(n).normal(0, 1, (2, n)).astype(np.float32)
    got = og.points_affect_points_vjp_self(og.Points(x, y, r, s), lu, lv, og.ExecEnv(og.CORE_GAUSSIAN, accum, ctx))
    for a, b in zip(restatement.self_vjp(og.CORE_GAUSSIAN, x, y, r, s, lu, lv), got):
        assert rel_err(a, b) < tol


def test_moment_passes_match_one_sided(ctx):
    """Gradient and VJP over several passes of row blocks, bit-identical when repeated."""
    n = 230_001
    x, y, r, s = cloud(n, n, 0.0, 0.004)
    lu, lv = np.random.default_rng(n).normal(0, 1, (2, n)).astype(np.float32)
    env = og.ExecEnv(og.CORE_GAUSSIAN, og.COMPENSATED, ctx)

    def both():
        p = og.Points(x, y, r, s)
        og.points_affect_points(p, p, og.VELANDGRAD, env)
        return [p.u, p.v, *p.grad, *og.points_affect_points_vjp_self(p, lu, lv, env)]

    a, b = both(), both()
    try:
        ctx.set_kernel_variant(og.VARIANT_PACKED2)
        c = both()
    finally:
        ctx.set_kernel_variant(og.VARIANT_AUTO)
    for p, q, t in zip(a, b, c):
        assert np.array_equal(p, q)
        assert rel_err(t, p) < 2e-5


@pytest.mark.parametrize("res", [og.VELONLY, og.VELANDGRAD])
@pytest.mark.parametrize("n", [300, 9001])
def test_equal_host_targets_are_the_set_itself(ctx, restatement, res, n):
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-1, 1, (2, n)).astype(np.float32)
    r, s = np.full(n, 0.02, np.float32), rng.normal(0, 1 / np.sqrt(n), n).astype(np.float32)
    env = og.ExecEnv(og.CORE_GAUSSIAN, og.COMPENSATED, ctx)
    same = og.Points(x, y, r, s)
    og.points_affect_points(same, same, res, env)
    copy = og.Points(x, y, r)
    og.points_affect_points(og.Points(x, y, r, s), copy, res, env)
    assert np.array_equal(same.u, copy.u) and np.array_equal(same.v, copy.v)
    tx = x.copy()
    tx[-1] += 0.25                                   # the last of them elsewhere: two sets
    other = og.Points(tx, y, r)
    og.points_affect_points(og.Points(x, y, r, s), other, res, env)
    u, v, _ = restatement.points_affect_points(og.CORE_GAUSSIAN, 1, x, y, r, s, tx, y, r, fp64=True)
    assert rel_err(u, other.u) < 2e-6 and rel_err(v, other.v) < 2e-6      # the tolerance of the sums above
    assert rel_err(u[-1:], other.u[-1:]) < 1e-4

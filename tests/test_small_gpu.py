"""GPU tests of the one-launch sums of small sets (csrc/p2p_small.cu, p2p_small_res.cu, adjoint_small.cu) at the edges of
their eight- and four-target blocks and 256-thread strides, against the FP64 oracle and the tiled kernels."""
import numpy as np
import pytest

import omega2d_gb300 as og
from conftest import rel_err

pytestmark = pytest.mark.gpu

CORES = [og.CORE_RM, og.CORE_GAUSSIAN, og.CORE_V2, og.CORE_WL, og.CORE_V3, og.CORE_SINGULAR, og.CORE_COMPACT_EXP]


# the tolerances of the packed kernels' tests: FP32 pairs with compensated or plain sums
@pytest.mark.parametrize("core", CORES)
@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 2e-6), (og.PLAIN_F32, 2e-5)])
@pytest.mark.parametrize("thick", [True, False])
@pytest.mark.parametrize("ns,nt", [(1, 1), (31, 7), (255, 8), (257, 9), (8193, 17), (9000, 1001)])
def test_small_sum_matches_fp64(ctx, restatement, core, accum, tol, thick, ns, nt):
    rng = np.random.default_rng(ns + nt + core)
    sx, sy, tx, ty = [rng.uniform(-1, 1, k).astype(np.float32) for k in (ns, ns, nt, nt)]
    sr, tr = [rng.uniform(0.01, 0.04, k).astype(np.float32) for k in (ns, nt)]
    ss = rng.normal(0, 1 / np.sqrt(ns), ns).astype(np.float32)
    tx[0], ty[0], tr[0] = sx[0], sy[0], sr[0]                 # a coincident pair
    t = og.Points(tx, ty, tr if thick else None, u=np.full(nt, 0.5, np.float32))
    before = ctx.launches
    og.points_affect_points(og.Points(sx, sy, sr, ss), t, og.VELONLY, og.ExecEnv(core, accum, ctx), finalize=True,
                            fs=(1.0, -0.25))
    assert ctx.launches - before == 1
    u64, v64, _ = restatement.points_affect_points(core, 1, sx, sy, sr, ss, tx, ty, tr if thick else None, fp64=True,
                                                   tu=np.full(nt, 0.5), tv=np.zeros(nt))
    assert rel_err(1.0 + u64 / (2 * np.pi), t.u) < tol
    assert rel_err(-0.25 + v64 / (2 * np.pi), t.v) < tol


# every pair evaluates the same core forms as the generic tiled kernels; only the order of the sums differs
@pytest.mark.parametrize("core", CORES)
@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 2e-6), (og.PLAIN_F32, 2e-5)])
@pytest.mark.parametrize("res", [og.VELANDGRAD, og.VELANDVORT, og.VELANDSHEAR])
@pytest.mark.parametrize("ns,nt,thick", [(1, 1, False), (255, 3, True), (257, 5, False), (8200, 1001, True)])
def test_small_results_match_generic(ctx, core, accum, tol, res, ns, nt, thick):
    rng = np.random.default_rng(ns + nt + core)
    sx, sy, tx, ty = [rng.uniform(-1, 1, k).astype(np.float32) for k in (ns, ns, nt, nt)]
    sr, tr = [rng.uniform(0.02, 0.04, k).astype(np.float32) for k in (ns, nt)]
    ss = rng.normal(0, 1 / np.sqrt(ns), ns).astype(np.float32)
    outs = []
    try:
        for variant in (og.VARIANT_GENERIC, og.VARIANT_AUTO):
            ctx.set_kernel_variant(variant)
            t = og.Points(tx, ty, tr if thick else None)
            og.points_affect_points(og.Points(sx, sy, sr, ss), t, res, og.ExecEnv(core, accum, ctx), finalize=True)
            outs.append([t.u, t.v] + [a for a in (t.vort, t.shear) if a is not None] + list(t.grad or []))
    finally:
        ctx.set_kernel_variant(og.VARIANT_AUTO)
    for a, b in zip(*outs):
        assert rel_err(a, b) < tol


@pytest.mark.parametrize("core", CORES)
@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 1e-5), (og.PLAIN_F32, 1e-4)])    # as tests/test_adjoint_gpu.py
@pytest.mark.parametrize("ns,nt,thick", [(1, 1, False), (3, 255, True), (5, 257, False), (1001, 8200, True)])
def test_small_vjp_matches_generic(ctx, core, accum, tol, ns, nt, thick):
    rng = np.random.default_rng(ns + nt + core)
    sx, sy, tx, ty = [rng.uniform(-1, 1, k).astype(np.float32) for k in (ns, ns, nt, nt)]
    sr, tr = [rng.uniform(0.02, 0.04, k).astype(np.float32) for k in (ns, nt)]
    ss = rng.normal(0, 1 / np.sqrt(ns), ns).astype(np.float32)
    lu, lv = rng.normal(0, 1, (2, nt)).astype(np.float32)
    src, targ, env = og.Points(sx, sy, sr, ss), og.Points(tx, ty, tr if thick else None), og.ExecEnv(core, accum, ctx)
    outs = []
    try:
        for variant in (og.VARIANT_GENERIC, og.VARIANT_AUTO):
            ctx.set_kernel_variant(variant)
            outs.append([og.points_affect_points_vjp(src, targ, lu, lv, env),
                         og.points_affect_points_vjp_self(src, lu[:ns] if nt >= ns else np.resize(lu, ns),
                                                          lv[:ns] if nt >= ns else np.resize(lv, ns), env)])
    finally:
        ctx.set_kernel_variant(og.VARIANT_AUTO)
    for ga, gb in zip(*outs):
        for a, b in zip(ga, gb):
            assert rel_err(a, b) < tol

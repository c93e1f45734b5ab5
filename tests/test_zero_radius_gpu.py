"""GPU tests of the one-launch VJP gather and gradient-type sums (csrc/adjoint_small.cu, p2p_small_res.cu) with Gaussian
sources of radius 0: away from its centre such a core is the point vortex."""
import numpy as np
import pytest

import omega2d_gb300 as og
from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 1e-5), (og.PLAIN_F32, 1e-4)])    # as tests/test_adjoint_gpu.py
@pytest.mark.parametrize("thick", [False, True])
@pytest.mark.parametrize("every", [1, 7])
def test_vjp_of_sources_without_radius(ctx, restatement, accum, tol, thick, every):
    rng = np.random.default_rng(every)
    sx, sy = rng.uniform(-1, 1, (2, 1000)).astype(np.float32)
    px, py = rng.uniform(2, 3, (2, 300)).astype(np.float32)       # far from all of them
    sr, ss = np.full(1000, 0.02, np.float32), rng.normal(0, 1, 1000).astype(np.float32)
    sr[::every] = 0.0
    lu, lv = rng.normal(0, 1, (2, 300)).astype(np.float32)
    got = og.points_affect_points_vjp(og.Points(sx, sy, sr, ss), og.Points(px, py, np.zeros(300, np.float32) if thick else None),
                                      lu, lv, og.ExecEnv(og.CORE_GAUSSIAN, accum, ctx))
    want = restatement.probe_vjp(og.CORE_SINGULAR, sx, sy, sr, ss, px, py, lu, lv)
    for a, b in zip(want, got):
        assert np.isfinite(b).all() and rel_err(a, b) < tol


@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 2e-6), (og.PLAIN_F32, 2e-5)])    # as tests/test_small_gpu.py
@pytest.mark.parametrize("thick", [False, True])
@pytest.mark.parametrize("every", [1, 7])
@pytest.mark.parametrize("res", [og.VELANDGRAD, og.VELANDVORT, og.VELANDSHEAR])
def test_results_of_sources_without_radius(ctx, accum, tol, thick, every, res):
    rng = np.random.default_rng(every)
    sx, sy = rng.uniform(-1, 1, (2, 1000)).astype(np.float32)
    px, py = rng.uniform(2, 3, (2, 300)).astype(np.float32)
    sr, ss = np.full(1000, 0.02, np.float32), rng.normal(0, 1, 1000).astype(np.float32)
    sr[::every] = 0.0
    outs = []
    for core, variant in ((og.CORE_SINGULAR, og.VARIANT_GENERIC), (og.CORE_GAUSSIAN, og.VARIANT_AUTO)):
        try:
            ctx.set_kernel_variant(variant)
            t = og.Points(px, py, np.zeros(300, np.float32) if thick else None)
            og.points_affect_points(og.Points(sx, sy, sr, ss), t, res, og.ExecEnv(core, accum, ctx))
        finally:
            ctx.set_kernel_variant(og.VARIANT_AUTO)
        outs.append([t.u, t.v] + [a for a in (t.vort, t.shear) if a is not None] + list(t.grad or []))
    size = max(np.abs(a).max() for a in outs[0])          # the vorticity away from the sources is 0
    for a, b in zip(*outs):
        assert np.isfinite(b).all() and np.max(np.abs(a - b)) < tol * size

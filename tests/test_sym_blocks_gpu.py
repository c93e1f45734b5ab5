"""GPU tests of the pair-once velocity sums (csrc/p2p_sym.cuh) past the one-launch kernel's range, at the edges of their
1024-row blocks (below 30,000 particles) and 2048-row blocks, every core in both accumulations against the FP64 oracle."""
import numpy as np
import pytest

import omega2d_gb300 as og
from conftest import rel_err

pytestmark = pytest.mark.gpu

CORES = [og.CORE_RM, og.CORE_GAUSSIAN, og.CORE_V2, og.CORE_WL, og.CORE_V3, og.CORE_SINGULAR, og.CORE_COMPACT_EXP]

SORTED = {og.CORE_GAUSSIAN: 25_000, og.CORE_COMPACT_EXP: 18_000}


# a block's last row and one over, one row over a 32-column group, an odd remainder; the first sizes of either kind
@pytest.mark.parametrize("core", CORES)
@pytest.mark.parametrize("spread", [0.0, 0.5])
@pytest.mark.parametrize("n", [6709, 7168, 7169, 8225, 9999, 17_999, 18_000, 24_999, 25_000, 30_000, 30_720, 30_721,
                               32_769])
def test_velocity_at_block_edges(ctx, restatement, core, spread, n):
    rng = np.random.default_rng(n + core)
    x, y = rng.uniform(-1, 1, (2, n)).astype(np.float32)
    r = (0.02 * rng.uniform(1 - spread, 1 + spread, n)).astype(np.float32)
    s = rng.normal(0, 1 / np.sqrt(n), n).astype(np.float32)
    x[5], y[5] = x[0], y[0]            # coincident particles, in one block and in two
    x[n - 1], y[n - 1] = x[1], y[1]
    k = np.unique(np.r_[:34, 1022:1026, 2046:2050, n // 2:n // 2 + 34, n - 34:n])
    u, v, _ = restatement.points_affect_points(core, 1, x, y, r, s, x[k], y[k], r[k], fp64=True, tu=np.full(k.size, 0.5),
                                               tv=np.zeros(k.size))
    # the tolerances of the packed kernels' tests: FP32 pairs with compensated or plain sums
    for accum, tol in ((og.COMPENSATED, 2e-6), (og.PLAIN_F32, 2e-5)):
        p = og.Points(x, y, r, s, u=np.full(n, 0.5, np.float32))
        before = ctx.launches
        og.points_affect_points(p, p, og.VELONLY, og.ExecEnv(core, accum, ctx), finalize=True, fs=(1.0, -0.25))
        # packing, sums, reduction; eight for the sort
        assert ctx.launches - before == (11 if n >= SORTED.get(core, n + 1) else 3)
        assert rel_err(1.0 + u / (2 * np.pi), p.u[k]) < tol and rel_err(-0.25 + v / (2 * np.pi), p.v[k]) < tol


# sorted from 3e8 pairs (eight launches more), in ranges of two units or more
@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 2e-6), (og.PLAIN_F32, 2e-5)])    # as tests/test_sym_gpu.py
@pytest.mark.parametrize("res", [og.VELANDGRAD, og.VELANDVORT, og.VELANDSHEAR])
@pytest.mark.parametrize("n,launches", [(17_320, 3), (17_321, 11), (28_545, 11)])
def test_results_about_the_spatial_order(ctx, accum, tol, res, n, launches):
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-1, 1, (2, n)).astype(np.float32)
    r, s = np.full(n, 0.02, np.float32), rng.normal(0, 1 / np.sqrt(n), n).astype(np.float32)
    outs = []
    try:
        for variant in (og.VARIANT_GENERIC, og.VARIANT_AUTO):
            ctx.set_kernel_variant(variant)
            p = og.Points(x, y, r, s)
            before = ctx.launches
            og.points_affect_points(p, p, res, og.ExecEnv(og.CORE_GAUSSIAN, accum, ctx), finalize=True)
            outs.append([p.u, p.v] + [a for a in (p.vort, p.shear) if a is not None] + list(p.grad or []))
    finally:
        ctx.set_kernel_variant(og.VARIANT_AUTO)
    assert ctx.launches - before == launches
    for a, b in zip(*outs):
        assert rel_err(a, b) < tol

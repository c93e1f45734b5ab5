"""GPU tests of the lines between the one-launch kernels and the tiled ones (csrc/adjoint_small.cu, p2p_small.cu,
p2p_small_res.cu) and of the tiled gathers' splits: which of them a call takes, by its launches, and its result against
the FP64 oracle."""
import numpy as np
import pytest

import omega2d_gb300 as og
from conftest import rel_err

pytestmark = pytest.mark.gpu


def points(n, seed):
    rng = np.random.default_rng(seed)
    x, y = rng.uniform(-1, 1, (2, n)).astype(np.float32)
    return x, y, np.full(n, 0.02, np.float32), rng.normal(0, 1 / np.sqrt(n), n).astype(np.float32)


def probe_vjp(ctx, core, accum, no, ne, seed):
    """Gradients, their oracle's at the first, last and some other sources (a source's need no other), and launches."""
    x, y, r, s = points(no, seed)
    px, py, _, _ = points(ne, seed + 1)
    lu, lv = np.random.default_rng(seed + 2).normal(0, 1, (2, ne)).astype(np.float32)
    before = ctx.launches
    got = og.points_affect_points_vjp(og.Points(x, y, r, s), og.Points(px, py), lu, lv, og.ExecEnv(core, accum, ctx))
    k = np.unique(np.r_[:8, no - 8:no, np.linspace(0, no - 1, 24).astype(int)].clip(0, no - 1))
    return [g[k] for g in got], (x[k], y[k], r[k], s[k], px, py, lu, lv), ctx.launches - before


# the tolerances of tests/test_adjoint_packed_gpu.py
@pytest.mark.parametrize("core", [og.CORE_GAUSSIAN, og.CORE_V2])
@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 1e-5), (og.PLAIN_F32, 1e-4)])
@pytest.mark.parametrize("no,ne,small", [(8, 30_000, True), (8, 140_000, False), (100, 300_001, False)])
def test_few_owners_many_elements(ctx, restatement, core, accum, tol, no, ne, small):
    got, args, launches = probe_vjp(ctx, core, accum, no, ne, no + ne)
    assert (launches == 1) == small
    for a, b in zip(restatement.probe_vjp(core, *args), got):
        assert rel_err(a, b) < tol


# one split; splits of one tile; a shorter last split; a second wave of blocks; more splits than one thread unrolls
@pytest.mark.parametrize("core", [og.CORE_GAUSSIAN, og.CORE_V2])
@pytest.mark.parametrize("no,ne", [(40_000, 200), (33_001, 812), (80_590, 812), (100_000, 1500), (70_000, 4500), (26_000, 4500),
                                   (17_000, 7001)])
def test_gather_splits(ctx, restatement, core, no, ne):
    got, args, launches = probe_vjp(ctx, core, og.COMPENSATED, no, ne, no + ne)
    assert launches > 1
    for a, b in zip(restatement.probe_vjp(core, *args), got):
        assert rel_err(a, b) < 1e-5


@pytest.mark.parametrize("core", [og.CORE_GAUSSIAN, og.CORE_V2])
@pytest.mark.parametrize("res,ns,nt,small", [(og.VELONLY, 32_768, 2400, True), (og.VELONLY, 20_000, 2500, True),
                                             (og.VELONLY, 20_001, 2500, False), (og.VELANDGRAD, 32_768, 1200, True),
                                             (og.VELANDGRAD, 28_001, 1300, False), (og.VELANDGRAD, 1000, 17_000, False),
                                             (og.VELANDVORT, 32_768, 1300, True)])
def test_one_launch_sums_past_a_wave(ctx, restatement, core, res, ns, nt, small):
    x, y, r, s = points(ns, ns + nt)
    tx, ty, _, _ = points(nt, nt)
    t = og.Points(tx, ty)
    before = ctx.launches
    og.points_affect_points(og.Points(x, y, r, s), t, res, og.ExecEnv(core, og.COMPENSATED, ctx))
    assert (ctx.launches - before == 1) == small
    k = np.r_[:16, nt - 16:nt]
    u, v, _ = restatement.points_affect_points(core, 1, x, y, r, s, tx[k], ty[k], None, fp64=True)
    assert rel_err(u, t.u[k]) < 2e-6 and rel_err(v, t.v[k]) < 2e-6


# the spatial order's lines in pairs and in targets, from just below
@pytest.mark.parametrize("core,sorts", [(og.CORE_GAUSSIAN, True), (og.CORE_COMPACT_EXP, False)])   # as the packed forms
@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 2e-6), (og.PLAIN_F32, 2e-5)])
@pytest.mark.parametrize("res", [og.VELANDGRAD, og.VELANDVORT, og.VELANDSHEAR])
@pytest.mark.parametrize("ns,nt,order", [(17_320, 17_320, False), (17_321, 17_321, True), (80_000, 4095, False),
                                         (80_000, 4096, True), (200_000, 3499, False), (200_000, 3500, True)])
def test_results_of_two_sets_about_the_spatial_order(ctx, core, sorts, accum, tol, res, ns, nt, order):
    x, y, r, s = points(ns, ns)
    tx, ty, _, _ = points(nt, nt + 1)
    outs, launches = [], []
    try:
        for by_name in (og.ORDER_INPUT, og.ORDER_AUTO):
            ctx.set_target_order(by_name)
            t = og.Points(tx, ty)
            before = ctx.launches
            og.points_affect_points(og.Points(x, y, r, s), t, res, og.ExecEnv(core, accum, ctx))
            launches.append(ctx.launches - before)
            outs.append([t.u, t.v] + [a for a in (t.vort, t.shear) if a is not None] + list(t.grad or []))
    finally:
        ctx.set_target_order(og.ORDER_AUTO)
    assert (launches[1] > launches[0]) == (order and sorts)
    for a, b in zip(*outs):
        assert rel_err(a, b) < tol


# plain sums: the one-launch kernels hold more blocks per SM and stay ahead further than the compensated ones
@pytest.mark.parametrize("core", [og.CORE_GAUSSIAN, og.CORE_V2, og.CORE_RM])
@pytest.mark.parametrize("res,ns,nt,small", [(og.VELONLY, 32_768, 2700, True), (og.VELONLY, 32_769, 2700, False),
                                             (og.VELANDGRAD, 32_768, 1373, True), (og.VELANDGRAD, 2197, 20_480, True),
                                             (og.VELANDGRAD, 2000, 20_481, False)])
def test_one_launch_plain_sums(ctx, restatement, core, res, ns, nt, small):
    x, y, r, s = points(ns, ns + nt)
    tx, ty, _, _ = points(nt, nt)
    t = og.Points(tx, ty)
    before = ctx.launches
    og.points_affect_points(og.Points(x, y, r, s), t, res, og.ExecEnv(core, og.PLAIN_F32, ctx))
    assert (ctx.launches - before == 1) == small
    k = np.r_[:16, nt - 16:nt]
    u, v, _ = restatement.points_affect_points(core, 1, x, y, r, s, tx[k], ty[k], None, fp64=True)
    assert rel_err(u, t.u[k]) < 2e-5 and rel_err(v, t.v[k]) < 2e-5


@pytest.mark.parametrize("core", [og.CORE_GAUSSIAN, og.CORE_V2])
@pytest.mark.parametrize("no,ne,small", [(8, 131_072, True), (8, 131_073, False), (3, 65_536, True), (3, 65_537, False),
                                         (24_576, 1500, True), (33_000, 1500, False)])
def test_one_launch_plain_gathers(ctx, restatement, core, no, ne, small):
    got, args, launches = probe_vjp(ctx, core, og.PLAIN_F32, no, ne, no + ne)
    assert (launches == 1) == small
    for a, b in zip(restatement.probe_vjp(core, *args), got):
        assert rel_err(a, b) < 1e-4

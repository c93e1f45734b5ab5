"""GPU tests of sets in spatial order whose radii vary: column groups beyond the largest radius' reach take the core's far
form (csrc/p2p_sym.cuh, sym_moments.cuh, p2p_packed_res.cu); against the generic kernels."""
import numpy as np
import pytest

import omega2d_gb300 as og
from conftest import rel_err

pytestmark = pytest.mark.gpu

KINDS = ["spread", "negative", "outlier", "nan"]


def radii(kind, n, rng):
    r = (0.01 * rng.uniform(0.6, 1.4, n)).astype(np.float32)
    if kind == "negative":
        r[::7] *= -2                    # the largest bit patterns, of radii that are not the largest
        r[3] = 0.5
    elif kind == "outlier":
        r[n // 2] = 0.7
    elif kind == "nan":
        r[n // 3] = np.nan
    return r


def both(ctx, fn):
    out = []
    try:
        for variant in (og.VARIANT_GENERIC, og.VARIANT_AUTO):
            ctx.set_kernel_variant(variant)
            out.append(fn())
    finally:
        ctx.set_kernel_variant(og.VARIANT_AUTO)
    return out


def check(pair, tol):
    for a, b in zip(*pair):
        assert np.array_equal(np.isnan(a), np.isnan(b))
        if not np.isnan(a).any():
            assert rel_err(a, b) < tol


def points(n, kind, seed):
    rng = np.random.default_rng(seed)
    x, y = rng.uniform(-1, 1, (2, n)).astype(np.float32)
    return x, y, radii(kind, n, rng), rng.normal(0, 1 / np.sqrt(n), n).astype(np.float32)


def outputs(p):
    return [p.u, p.v] + [a for a in (p.vort, p.shear) if a is not None] + list(p.grad or [])


# tolerances as in tests/test_sym_gpu.py and tests/test_adjoint_packed_gpu.py
@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 2e-6), (og.PLAIN_F32, 2e-5)])
@pytest.mark.parametrize("core,n", [(og.CORE_GAUSSIAN, 26_001), (og.CORE_GAUSSIAN, 64_007), (og.CORE_COMPACT_EXP, 18_500)])
@pytest.mark.parametrize("kind", KINDS)
def test_velocity(ctx, core, n, accum, tol, kind):
    def run():
        p = og.Points(*points(n, kind, n))
        og.points_affect_points(p, p, og.VELONLY, og.ExecEnv(core, accum, ctx))
        return outputs(p)
    check(both(ctx, run), tol)


@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 2e-6), (og.PLAIN_F32, 2e-5)])
@pytest.mark.parametrize("res", [og.VELANDGRAD, og.VELANDVORT, og.VELANDSHEAR])
@pytest.mark.parametrize("kind", KINDS)
def test_results(ctx, res, accum, tol, kind):
    def run():
        p = og.Points(*points(17_400, kind, 1))
        og.points_affect_points(p, p, res, og.ExecEnv(og.CORE_GAUSSIAN, accum, ctx))
        return outputs(p)
    check(both(ctx, run), tol)


@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 2e-6), (og.PLAIN_F32, 2e-5)])
@pytest.mark.parametrize("res", [og.VELANDGRAD, og.VELANDVORT, og.VELANDSHEAR])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("thick", [False, True])
def test_results_of_two_sets(ctx, res, accum, tol, kind, thick):
    def run():
        s = og.Points(*points(17_400, kind, 2))
        x, y, r, g = points(17_301, "spread", 3)
        t = og.Points(x, y, r, g) if thick else og.Points(x, y)
        og.points_affect_points(s, t, res, og.ExecEnv(og.CORE_GAUSSIAN, accum, ctx))
        return outputs(t)
    check(both(ctx, run), tol)


@pytest.mark.parametrize("accum,tol", [(og.COMPENSATED, 1e-5), (og.PLAIN_F32, 1e-4)])
@pytest.mark.parametrize("kind", KINDS)
def test_vjp(ctx, accum, tol, kind):
    lu, lv = np.random.default_rng(4).normal(0, 1, (2, 26_500)).astype(np.float32)

    def run():
        p = og.Points(*points(26_500, kind, 5))
        return og.points_affect_points_vjp_self(p, lu, lv, og.ExecEnv(og.CORE_GAUSSIAN, accum, ctx))
    check(both(ctx, run), tol)

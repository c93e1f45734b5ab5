"""The far form of the panel sums (csrc/panels.cu, pan_far_inverse): its truncated series against the exact functions
on the CPU, and both panel sums with every target on one side of its limit, at the limit and beyond, on the GPU."""
import numpy as np
import pytest

import omega2d_gb300 as og
from conftest import rel_err

FAR = 3163.0        # |z - m|^2 > FAR |h|^2


def test_far_series_matches_log():
    """log((z - z0)/(z - z1)) = 2 (q + q^3/3) + O(q^5), q = h/(z - m): the next term is below 2e-8 relative there, and
    the kernel's arrangement (A + i B = -1/conj(z - m), n + i m = (A + i B)^2 with n = 2 A^2 - 1/d2) is that series."""
    rng = np.random.default_rng(0)
    h = 10.0 ** rng.uniform(-4, 0, 4000) * np.exp(2j * np.pi * rng.uniform(0, 1, 4000))
    d = np.abs(h) * np.sqrt(FAR) * 10.0 ** rng.uniform(0, 3, 4000) * np.exp(2j * np.pi * rng.uniform(0, 1, 4000))
    exact = 2.0 * np.arctanh(h / d)
    d2 = np.abs(d) ** 2
    A, B = -d.real / d2, -d.imag / d2
    p2 = (2.0 * A * A - 1.0 / d2) + 1j * (2.0 * A * B)
    g = 1.7 - 0.3j
    d1, d3 = -2.0 * np.conj(g * h), -(2.0 / 3.0) * np.conj(g * h ** 3)
    got = np.conj((A + 1j * B) * (d1 + d3 * p2))
    assert np.max(np.abs(got - g * exact) / np.abs(g * exact)) < 2.1e-8


@pytest.mark.gpu
@pytest.mark.parametrize("ring", [0.5, 0.99, 1.01, 8.0])
@pytest.mark.parametrize("npan,n", [(31, 300), (130, 4097)])
@pytest.mark.parametrize("accum,tol", [(og.PLAIN_F32, 5e-5), (og.COMPENSATED, 2e-5)])   # as tests/test_panels_gpu.py
def test_far_form_edges(ctx, restatement, ring, npan, n, accum, tol):
    """A short row of panels near (0.3, -0.2) and points on a ring at `ring` times the far limit of every panel."""
    rng = np.random.default_rng(npan + n)
    h = 0.002
    nodes = np.arange(npan + 1)
    bx = (0.3 + 0.02 * h * nodes).astype(np.float32)           # panels 0.02 h apart, each 2 h long and tilted
    idx = np.stack([2 * np.arange(npan), 2 * np.arange(npan) + 1], 1).ravel()
    nx = np.stack([bx[:-1] - h, bx[:-1] + h], 1).ravel()
    ny = np.stack([np.full(npan, -0.2 - 0.3 * h), np.full(npan, -0.2 + 0.3 * h)], 1).ravel()
    half = h * np.hypot(1.0, 0.3)
    body = og.Surfaces(nx, ny, idx, vs=rng.normal(0, 1, npan), ss=rng.normal(0, 1, npan))
    a = rng.uniform(0, 2 * np.pi, n)
    rad = ring * half * np.sqrt(FAR) + (0.02 * h * npan if ring > 1 else 0.0)
    x = (0.3 + 0.01 * h * npan + rad * np.cos(a)).astype(np.float32)
    y = (-0.2 + rad * np.sin(a)).astype(np.float32)
    s = rng.normal(0, 1, n).astype(np.float32)
    env = og.ExecEnv(accum=accum, context=ctx)
    t = og.Points(x, y)
    og.panels_affect_points(body, t, env)
    u, v = restatement.panels_affect_points(body.nx, body.ny, body.idx, body.vs, body.ss, x, y, fp64=True)
    assert rel_err(np.hypot(u, v), np.hypot(t.u, t.v)) < tol
    og.points_affect_panels(og.Points(x, y, np.full(n, 0.01, np.float32), s), body, env)
    u, v = restatement.points_affect_panels(x, y, s, body.nx, body.ny, body.idx, fp64=True)
    assert rel_err(u, body.pu) < tol and rel_err(v, body.pv) < tol

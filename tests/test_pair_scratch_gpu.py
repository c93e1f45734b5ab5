"""GPU tests of the pair-once sums short of device memory (csrc/p2p_sym.cu, sym_moments.cu): a limit on their work buffer
stands in for a full device.  They go through more passes and, below one row block at a time, leave the sum to the
one-sided kernels, which keep the buffer that is there."""
import numpy as np
import pytest

import omega2d_gb300 as og
from conftest import rel_err

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture
def own():
    c = og.Context(0)
    yield c
    c.close()


def run(c, n, core, res):
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-1, 1, (2, n)).astype(np.float32)
    r, s = np.full(n, 0.01, np.float32), rng.normal(0, 1 / np.sqrt(n), n).astype(np.float32)
    env, before = og.ExecEnv(core, og.COMPENSATED, c), c.launches
    p = og.Points(x, y, r, s)
    if res == "vjp":
        lu, lv = rng.normal(0, 1, (2, n)).astype(np.float32)
        out = list(og.points_affect_points_vjp_self(p, lu, lv, env))
    else:
        og.points_affect_points(p, p, res, env)
        out = [p.u, p.v] + list(p.grad or [])
    return out, c.launches - before


# launches: packing (and eight for the sort), then two a pass
@pytest.mark.parametrize("n,core,res,first,limits", [(70_000, og.CORE_V2, og.VELONLY, 1, (30, 15, 2)),
                                                     (40_000, og.CORE_GAUSSIAN, og.VELANDGRAD, 9, (60, 30, 2)),
                                                     (40_000, og.CORE_GAUSSIAN, "vjp", 9, (40, 20, 2))])
def test_short_of_memory(own, n, core, res, first, limits):
    full, launches = run(own, n, core, res)
    assert launches == first + 2
    passes = [1]
    for mb in limits[:2]:
        own.selftest_pair_scratch(mb * MB)
        got, launches = run(own, n, core, res)
        passes.append((launches - first) // 2)
        assert launches == first + 2 * passes[-1]
        for a, b in zip(full, got):
            assert rel_err(a, b) < 2e-6
    assert passes[0] < passes[1] < passes[2]
    own.set_kernel_variant(og.VARIANT_PACKED2)       # one-sided by name
    _, one_sided = run(own, n, core, res)
    own.set_kernel_variant(og.VARIANT_AUTO)
    own.selftest_pair_scratch(limits[2] * MB)
    for _ in range(2):                               # and again with what the first one left
        got, launches = run(own, n, core, res)
        assert launches == one_sided
        for a, b in zip(full, got):
            assert rel_err(a, b) < 2e-5              # one-sided against pair-once gradients, as tests/test_sym_gpu.py
    own.selftest_pair_scratch(0)
    again, launches = run(own, n, core, res)
    assert launches == first + 2
    for a, b in zip(full, again):
        assert np.array_equal(a, b)

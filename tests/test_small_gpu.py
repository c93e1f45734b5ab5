"""GPU tests of the one-launch velocity sum of small sets (csrc/p2p_small.cu) at the edges of its eight-target blocks and
256-thread strides, against the FP64 oracle, for every core."""
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

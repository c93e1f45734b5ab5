"""GPU test of the fused GMRES cycle on systems whose row groups form one thread-block cluster (csrc/gmres.cu: two to
sixteen groups of 32 rows) and just beyond, with last groups of one row and of 31."""
import numpy as np
import pytest

import omega2d_gb300 as og

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 63, 97, 480, 481, 511, 512, 513])
def test_cluster_cycle(n):
    rng = np.random.default_rng(n)
    A = np.eye(n) + 0.3 * rng.normal(0, 1 / np.sqrt(n), (n, n))
    b = rng.normal(0, 1, n)
    c = og.Context()
    try:
        x, it, rel = og.solve_gmres_f64(A, b, tol=1e-12, restart=50, context=c)
        x2, it2, _ = og.solve_gmres_f64(A, b, tol=1e-12, restart=50, context=c)
    finally:
        c.close()
    assert it == it2 and np.array_equal(x, x2)             # every sum has a fixed order
    assert np.linalg.norm(b - A @ x) <= 1.01e-12 * np.linalg.norm(b)     # the tolerance asked for, and its rounding

"""FP64 handles of a few particles: the once-per-pair kernels walk live sources
only and finish a single block themselves.

Values: against the all-pairs kernels, which sum the same FP64 terms: 1e-12.
Time: one particle has one pair term to evaluate, 32 have 32; a walk over all 32
slots took the same for both.  The kernels are FP64-issue bound, so one particle
is to take at most three quarters of the time of 32 (launches included).
"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def handle(mf, n, sym):
    rng = np.random.default_rng(n)
    pos = rng.random((n, 3)).astype(np.float32)
    s = mf.Solver(n, 0.5, 0.5, 0.05, 0.5, (0.0, 0.3, 1.0), None, None, pos, precision="fp64")
    s.set_option("solver", mf.SOLVER_CG)
    s.set_option("pair_symmetric", sym)
    s.solve(50)
    s.evaluate_fitted_near_foece()
    return s


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 40, 63, 64, 65, 96])
def test_values(mf, cuda, n):
    out = []
    for sym in (0, 1):
        s = handle(mf, n, sym)
        m = np.random.default_rng(1).normal(size=(n, 3)).astype(np.float32)
        out.append((s.apply_field(m), s.get("magnetic_bodyforce", f64=True), s.get("total_B_over_mu0", f64=True)))
        s.close()
    for a, b in zip(*out):
        assert np.abs(np.asarray(a, float) - b).max() <= 1e-12 * max(np.abs(np.asarray(out[0][2], float)).max(), np.abs(b).max())


def test_time(mf, cuda):
    t = []
    for n in (1, 32):
        s = handle(mf, n, 1)
        r = []
        for _ in range(30):
            t0 = time.perf_counter()
            s.evaluate_fitted_near_foece()
            r.append(time.perf_counter() - t0)
        t.append(min(r))
        s.close()
    assert t[0] < 0.75 * t[1]

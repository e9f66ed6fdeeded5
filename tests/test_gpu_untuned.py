"""The default block shapes of untuned handles (MF_OPT_AUTOTUNE 0): the packed force
of one scene runs once per unordered pair only from the size on where that has
block pairs enough, and both sides give the oracle's force.

Tolerance: the FP32 kernels' stated bar, relative L2 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,once", [(8192, False), (10001, False), (13311, False), (13312, True), (16384, True)])
def test_force(mf, cuda, oracle, n, once):
    import scenes
    sc = scenes.jittered_lattice(n, "sphere", chi=2.0, seed=n)
    s = mf.Solver(n, sc.h, sc.h, sc.volume, 0.1, sc.H0, None, None, sc.pos)
    for k, v in (("solver", mf.SOLVER_CG), ("autotune", 0), ("pair_symmetric", 1), ("fused_products", 0), ("kernel_timing", 1)):
        s.set_option(k, v)
    s.solve(20)
    s.reset_counters()
    s.evaluate_fitted_near_foece()
    k = s.kernel_stats("force")
    assert (k["evals"] < k["pairs"]) == once
    m = s.get("M").astype(np.float64)
    i = np.random.default_rng(1).choice(n, 64, replace=False)
    pd = sc.pos.astype(np.float64)
    want = np.einsum("icr,ic->ir", oracle.tensor_sum(pd[i], pd, m, float(np.float32(sc.h))).reshape(-1, 3, 3), m[i])
    got = s.get("magnetic_bodyforce")[i].astype(np.float64)
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < 1e-5
    s.close()

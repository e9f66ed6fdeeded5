"""The once-per-pair kernels where the items' rotation over the lanes can go
wrong: last tiles of one particle, of a whole group of 32 items and one more or
less, and of an odd count; the separate products and both in one launch, against
the all-pairs kernels and the FP64 oracle.

Tolerances: the same FP32 pair terms in another order, 2e-6 between the kernels
(as tests/test_gpu_fused.py); the FP32 bar against the oracle, 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def products(mf, pos, h, vol, sym, fused):
    s = mf.Solver(len(pos), h, h, vol, 1.5, (0.0, 0.0, 1.0), None, None, pos)
    s.set_option("pair_symmetric", sym)
    s.set_option("fmm", mf.FMM_OFF)
    s.set_option("solver", mf.SOLVER_CG)
    s.set_option("rel_tol", 3e-7)
    s.solve(200)
    s.set_option("rel_tol", 1e-6)
    s.set_option("fused_products", fused)
    s.set_option("kernel_timing", 1)
    s.reset_counters()
    s.solve(200)  # the warm start stands: b is unchanged
    s.evaluate_fitted_near_foece()
    out = s.total_B_over_mu0, s.M, s.magnetic_bodyforce, {k: s.kernel_stats(k) for k in ("force", "field_force")}
    s.close()
    return out


@pytest.mark.parametrize("n", [14336 + 1, 14336 + 62, 14336 + 64, 14336 + 65, 15 * 1024 + 513, 16 * 1024 - 1])
def test_last_tiles(mf, cuda, oracle, n):
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    pos = ((g + 0.4 * rng.random(g.shape)) / side).astype(np.float32)
    h, vol = 2.0 / side, 1.0 / side ** 3
    b0, m0, f0, _ = products(mf, pos, h, vol, 0, 0)
    b1, m1, f1, k1 = products(mf, pos, h, vol, 2, 0)
    b2, m2, f2, k2 = products(mf, pos, h, vol, 2, 2)
    assert k1["force"]["evals"] < k1["force"]["pairs"] and k2["field_force"]["launches"] == 1
    assert rel(b1, b0) < 2e-6 and rel(b2, b0) < 2e-6
    idx = np.r_[0:32, n - 32:n, rng.choice(n, 64, replace=False)]
    pd = pos.astype(np.float64)
    for m, f in ((m0, f0), (m1, f1), (m2, f2)):
        md = np.asarray(m, np.float64)
        T = oracle.tensor_sum(pd[idx], pd, md, float(np.float32(h))).reshape(-1, 3, 3)
        assert rel(f[idx], np.einsum("icr,ic->ir", T, md[idx])) < 1e-5
    # the last tile's own field: residual of the fixed point at its particles
    c = vol * 1.5 / 2.5
    want = oracle.field(pd[idx], pd, c * np.asarray(b2, np.float64), float(np.float32(h))) + [0.0, 0.0, 1.0]
    assert rel(b2[idx], want) < 1e-5

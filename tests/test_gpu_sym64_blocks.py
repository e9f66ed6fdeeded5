"""FP64 products once per unordered pair at every block size, up to the largest
(eight warps a block, from 32,768 particles on), against the all-pairs kernels.

Values: both sum the same FP64 terms, the field read back in FP32: 1e-6 of the
largest; the forces of one and the same magnetization 1e-11.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8192, 16384, 32767, 32768, 32769, 40001])
def test_against_all_pairs(mf, cuda, n):
    rng = np.random.default_rng(n)
    pos = rng.random((n, 3)).astype(np.float32)
    pos[n - 1] = pos[0]  # a coincident pair across blocks
    m = rng.normal(size=(n, 3)).astype(np.float32)
    v = 1.0 / n
    out = []
    for sym in (0, 1):
        s = mf.Solver(n, 2 * v ** (1 / 3), 0.1, v, 0.05, (0.0, 0.3, 1.0), None, None, pos, precision="fp64")
        for k, x in (("pair_symmetric", sym), ("solver", mf.SOLVER_CG), ("rel_tol", 1e-3), ("kernel_timing", 1)):
            s.set_option(k, x)
        f = s.apply_field(m).astype(float)
        k = s.kernel_stats("field")
        assert (k["evals"] < k["pairs"]) == bool(sym)
        s.solve(1)
        s.evaluate_fitted_near_foece()
        out.append((f, s.get("total_B_over_mu0", f64=True), s.get("magnetic_bodyforce", f64=True)))
        s.close()
    (f0, b0, F0), (f1, b1, F1) = out
    assert np.abs(f1 - f0).max() <= 1e-6 * np.abs(f0).max()
    assert np.linalg.norm(b1 - b0) <= 1e-12 * np.linalg.norm(b0)
    assert np.linalg.norm(F1 - F0) <= 1e-11 * np.linalg.norm(F0)

"""FP64 products once per unordered pair, where they can go wrong: block and
warp remainders, one block, each block size, coincident particles, and
distances exactly on the near radii and the fitted curves' joins.

Tolerances.  Both FP64 kernels sum the same pair terms in FP64; a pair term
differs by a few roundings (1e-15), and solves to 1e-13 may stop one iteration
apart: 1e-11 between the kernels.  Against the FP64 oracle the stated bar of
the FP64 path, 1e-8.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def solved(mf, pos, h, vol, chi, sym):
    n = len(pos)
    s = mf.Solver(n, h, h, vol, chi, (0.0, 0.3, 1.0), None, None, pos, precision="fp64")
    s.set_option("pair_symmetric", 1 if sym else 0)
    s.set_option("solver", mf.SOLVER_CG)
    s.set_option("rel_tol", 1e-13)
    s.set_option("kernel_timing", 1)
    s.solve(300)
    s.evaluate_fitted_near_foece()
    k = s.kernel_stats("field")
    out = s.get("total_B_over_mu0", f64=True), s.get("magnetic_bodyforce", f64=True), k
    s.close()
    return out


def check(mf, pos, h, vol, chi):
    b0, f0, k0 = solved(mf, pos, h, vol, chi, False)
    b1, f1, k1 = solved(mf, pos, h, vol, chi, True)
    if len(pos) > 1:  # the once-per-pair kernel ran
        assert k0["evals"] == k0["pairs"] and k1["evals"] < k1["pairs"]
    assert rel(b1, b0) < 1e-11
    scale = max(np.linalg.norm(f0), 1e-300)
    # forces that cancel by symmetry (one particle, a lattice) are compared on
    # the scale of one pair's force at distance h
    pair = 3 * 1.25663706e-6 / (4 * np.pi) * (vol * chi / (1 + chi)) ** 2 / h ** 4
    assert np.linalg.norm(f1 - f0) < 1e-11 * max(scale, pair * np.sqrt(len(pos)))
    return b1, f1


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 65, 1000, 2047, 2048, 2049, 8191, 8193, 16385])
def test_sizes_against_all_pairs(mf, cuda, n):
    rng = np.random.default_rng(n)
    pos = rng.random((n, 3)).astype(np.float32)
    if n > 4:
        pos[1] = pos[0]  # a coincident pair
    vol = 1.0 / max(n, 64)
    check(mf, pos, 2 * vol ** (1 / 3), vol, 1.0)


def test_distances_on_the_joins(mf, cuda):
    # h = 2 spacings, spacing a power of two: r / h = 0.5, 1, 1.5, 2, .. 4 exactly
    g = np.arange(11, dtype=np.float32) * 0.125
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    check(mf, pos, 0.25, 0.125 ** 3, 1.0)


def test_against_the_oracle(mf, cuda, oracle):
    rng = np.random.default_rng(5)
    n, vol, chi = 700, 1.0 / 700, 1.2
    pos = rng.random((n, 3)).astype(np.float32)
    h = float(np.float32(2 * vol ** (1 / 3)))
    b, f = check(mf, pos, h, vol, chi)
    vol, chi = float(np.float32(vol)), float(np.float32(chi))
    c = vol * chi / (1 + chi)
    hext, _ = oracle.ext(pos, None, None, (0.0, float(np.float32(0.3)), 1.0), h)
    bo, _, _ = oracle.solve_cg(pos, h, c, hext, rel_tol=1e-13)
    assert rel(b, bo) < 1e-8
    assert rel(f, oracle.force(pos, c * bo, h)) < 1e-8

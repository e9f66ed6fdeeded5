"""The near-field corrections through entries that always take them, whatever the
size: separate targets through the FMM matrix (k_correction_at), one set through
handles whose packed products are forced (k_correction_cells).

Geometry: warp remainders, targets outside the sources' box and on its corners,
targets at sources, slabs, far clusters; cells of 1, 2, 7, 8, 9 and 17 particles,
empty cells, both numbers of warps per cell, coincident particles, lattices with
every distance on the near radii and the curves' joins (spacing a power of two,
h two spacings: exact in FP32).

Tolerance: the FP32 kernels' stated bar against the FP64 oracle, relative L2 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def sources(kind, ns, rng):
    if kind == "cube":
        return rng.random((ns, 3)).astype(np.float32)
    if kind == "slab":  # a flat grid: few cells along z
        return (rng.random((ns, 3)) * [1.0, 1.0, 0.01]).astype(np.float32)
    if kind == "lattice":  # distances exactly h/2, h, .. 4h at h = 1/8
        k = int(np.ceil(ns ** (1 / 3)))
        return (np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:ns] / 16).astype(np.float32)
    p = rng.random((ns, 3)) * 0.2  # two far clusters: most cells empty, cells widened
    p[ns // 2:, 0] += 40.0
    return p.astype(np.float32)


@pytest.mark.parametrize("kind", ["cube", "slab", "clusters", "lattice"])
@pytest.mark.parametrize("nt,ns,h", [(1, 900, 0.2), (5, 33, 0.5), (131, 4000, 0.03), (1000, 2999, 0.125)])
def test_separate_targets(mf, cuda, oracle, kind, nt, ns, h):
    rng = np.random.default_rng(nt + ns)
    s = sources(kind, ns, rng)
    lo, hi = s.min(axis=0), s.max(axis=0)
    t = (lo - 3 * h + rng.random((nt, 3)) * (hi - lo + 6 * h)).astype(np.float32)
    if kind == "lattice":
        t[:] = s[rng.integers(0, ns, nt)]
    k = max(1, nt // 8)
    t[:min(k, ns)] = s[:min(k, ns)]                      # at sources
    t[-k:] = np.where(rng.random((k, 3)) < 0.5, lo, hi)  # corners and edges of the box
    m = rng.normal(size=(ns, 3)).astype(np.float32)
    h = float(np.float32(h))
    A = mf.FmmMatrix(s, h, targets=t, order=8, theta=0.02)
    td, sd = t.astype(np.float64), s.astype(np.float64)
    assert rel(A.field(m), oracle.field(td, sd, m, h)) < TOL
    assert rel(A.hessian(m), oracle.tensor_sum(td, sd, m.astype(np.float64), h).reshape(-1, 9)) < TOL
    A.close()


def clumps(per, cells, h, rng):
    """`cells` clumps a side of `per` particles, h apart: cells of exactly that many."""
    g = np.stack(np.meshgrid(*[np.arange(cells)] * 3, indexing="ij"), -1).reshape(-1, 3)
    p = (g[:, None] + 0.5 + 0.3 * (rng.random((len(g), per, 3)) - 0.5)).reshape(-1, 3)
    return (p * h * 1.0001).astype(np.float32)


def products(mf, pos, m_scale, h):
    """Packed field of given dipoles, and the packed force of the handle's own."""
    n = len(pos)
    s = mf.Solver(n, h, h, 0.1 * h ** 3, 0.1, (0.2, -0.3, 1.0), None, None, pos)
    for k, v in (("solver", mf.SOLVER_CG), ("autotune", 0), ("pair_symmetric", 2), ("fused_products", 0), ("kernel_timing", 1)):
        s.set_option(k, v)
    m = (m_scale * np.random.default_rng(3).normal(size=(n, 3))).astype(np.float32)
    f = s.apply_field(m)
    k = s.kernel_stats("field")
    assert k["evals"] < k["pairs"]  # the packed field ran, with its correction
    s.solve(30)
    s.reset_counters()
    s.evaluate_fitted_near_foece()
    packed_force = s.kernel_stats("force")
    out = m, f, s.get("M"), s.get("magnetic_bodyforce"), packed_force["evals"] < packed_force["pairs"]
    s.close()
    return out


def check(oracle, pos, h, res, force):
    m, f, M, F, packed = res
    i = np.unique(np.r_[0:64, np.random.default_rng(1).choice(len(pos), 200), len(pos) - 16:len(pos)])
    pd = pos.astype(np.float64)
    assert rel(f[i], oracle.field(pd[i], pd, m, h)) < TOL
    assert packed == force
    T = oracle.tensor_sum(pd[i], pd, M.astype(np.float64), h).reshape(-1, 3, 3)
    assert rel(F[i], np.einsum("icr,ic->ir", T, M[i].astype(np.float64))) < TOL


@pytest.mark.parametrize("per,cells", [(1, 13), (2, 11), (7, 7), (8, 7), (9, 7), (17, 5),       # field: four warps a cell
                                       (1, 21), (2, 21), (7, 11), (9, 10), (17, 8)])            # and the force packed
def test_cells_of_every_fill(mf, cuda, oracle, per, cells):
    rng = np.random.default_rng(per)
    h = 0.0625
    pos = clumps(per, cells, h, rng)
    if per > 1:
        pos[1] = pos[0]
    check(oracle, pos, h, products(mf, pos, 1e-4, h), force=len(pos) >= 8192)


@pytest.mark.parametrize("side", [14, 24, 31])  # few cells; the force packed; one warp a cell
@pytest.mark.parametrize("jitter", [0.0, 0.3])
def test_lattices(mf, cuda, oracle, side, jitter):
    rng = np.random.default_rng(side)
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = ((g + jitter * rng.random(g.shape)) / 32).astype(np.float32)
    check(oracle, pos, 1 / 16, products(mf, pos, 1e-4, 1 / 16), force=len(pos) >= 8192)

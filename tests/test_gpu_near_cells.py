"""The packed near-field correction over cells against the FP64 oracle, where
its passes can go wrong: cells with one, seven, eight and nine particles (the
passes of eight targets and their last pair), empty cells, both warp counts,
coincident particles, and distances on the near radii and the curves' joins.

Tolerance: the FP32 kernels' stated bar against the oracle, relative L2 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


def clumps(per, cells, h, rng):
    """`cells` clumps of `per` particles, h apart: cells of exactly that many."""
    g = np.stack(np.meshgrid(*[np.arange(cells)] * 3, indexing="ij"), -1).reshape(-1, 3)
    p = (g[:, None] + 0.5 + 0.3 * (rng.random((len(g), per, 3)) - 0.5)).reshape(-1, 3)
    return (p * h * 1.0001).astype(np.float32)


@pytest.mark.parametrize("per,cells", [(1, 12), (2, 5), (7, 6), (8, 6), (9, 6), (17, 4)])
def test_cells_of_every_fill(mf, cuda, oracle, per, cells):
    rng = np.random.default_rng(per)
    h = 0.0625
    p = clumps(per, cells, h, rng)
    if per > 1:
        p[1] = p[0]
    m = rng.normal(size=p.shape).astype(np.float32)
    t, q = dev(cuda, p), dev(cuda, m)
    assert rel(mf.direct_field(t, t, q, h).cpu().numpy(), oracle.field(p, p, m, h)) < TOL
    assert rel(mf.direct_force(t, q, h).cpu().numpy(), oracle.force(p, m, h)) < TOL


@pytest.mark.parametrize("n", [9000, 70000])
def test_lattices_of_few_and_many_cells(mf, cuda, oracle, n):
    rng = np.random.default_rng(n)
    side = int(round(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    p = ((g + 0.3 * rng.random(g.shape)) / side).astype(np.float32)
    m = (rng.normal(size=p.shape) + [0, 0, 3]).astype(np.float32)
    h = 2.0 / side
    idx = rng.choice(len(p), 128, replace=False)
    t, q = dev(cuda, p), dev(cuda, m)
    f = mf.direct_force(t, q, h).cpu().numpy()[idx]
    b = mf.direct_field(t, t, q, h).cpu().numpy()[idx]
    pd, md = p.astype(np.float64), m.astype(np.float64)
    T = oracle.tensor_sum(pd[idx], pd, md, h).reshape(-1, 3, 3)
    assert rel(b, oracle.field(pd[idx], pd, md, h)) < TOL
    assert rel(f, np.einsum("icr,ic->ir", T, md[idx])) < TOL

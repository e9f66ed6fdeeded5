"""Targets concentrated in few leaf boxes of the FMM matrix, as of a field map of a
small region, and bodies of a dense and a thin part: values against the FP64
oracle, and the time against evenly spread targets.

Tolerance: the operator's stated bar at order 8, relative L2 1e-5.  Time: a
target inside the body has the same number of near sources wherever it is, so
concentrated ones are to take at most twice the time of spread ones.
"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


def rel(a, b):
    return np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b)


def best(f, n=9):
    f()
    t = []
    for _ in range(n):
        t0 = time.perf_counter()
        f()
        t.append(time.perf_counter() - t0)
    return min(t)


@pytest.mark.parametrize("where", ["box", "line"])
def test_time(mf, cuda, where):
    rng = np.random.default_rng(1)
    src = rng.random((150000, 3)).astype(np.float32)
    m = (rng.normal(size=src.shape) + [0, 0, 2]).astype(np.float32)
    u = rng.random((10000, 3))
    few = {"box": u * 0.05 + 0.5, "line": np.c_[u[:, :1], np.full((10000, 2), 0.43)]}[where]
    t = []
    for tgt in (u, few):
        A = mf.FmmMatrix(src, 2 * 150000 ** (-1 / 3), targets=tgt.astype(np.float32), order=8)
        t.append((best(lambda: A.field(m)), best(lambda: A.hessian(m))))
        A.close()
    assert t[1][0] < 2 * t[0][0] and t[1][1] < 2 * t[0][1]


@pytest.mark.parametrize("nt", [16, 17, 100, 4001])
def test_targets_in_one_box(mf, oracle, nt):
    rng = np.random.default_rng(nt)
    src = rng.random((20000, 3)).astype(np.float32)
    m = (rng.normal(size=src.shape) + [0, 0, 2]).astype(np.float32)
    tgt = (0.51 + 0.04 * rng.random((nt, 3))).astype(np.float32)
    A = mf.FmmMatrix(src, 0.05, targets=tgt, order=8, theta=0.5)
    k = np.unique(np.r_[0:min(nt, 20), max(0, nt - 20):nt])
    td, sd = tgt[k].astype(np.float64), src.astype(np.float64)
    assert rel(A.field(m)[k], oracle.field(td, sd, m, 0.05)) < TOL
    assert rel(A.hessian(m)[k], oracle.tensor_sum(td, sd, m.astype(np.float64), 0.05).reshape(-1, 9)) < TOL
    A.close()


def test_dense_and_thin_parts(mf, oracle):
    """Targets = sources: 6,000 particles in one leaf box, 14,000 over the others."""
    rng = np.random.default_rng(7)
    p = np.r_[rng.random((14000, 3)), 0.51 + 0.04 * rng.random((6000, 3))].astype(np.float32)
    m = (rng.normal(size=p.shape) + [0, 0, 2]).astype(np.float32)
    A = mf.FmmMatrix(p, 0.02, order=8)
    k = rng.choice(len(p), 200, replace=False)
    assert rel(A.field(m)[k], oracle.field(p[k].astype(np.float64), p.astype(np.float64), m, 0.02)) < TOL
    A.close()

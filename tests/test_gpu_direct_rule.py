"""Direct sums on both sides of the pair count where the packed kernels take
over from the exact-branch ones, odd counts and few targets or sources included,
against the FP64 oracle at a sample of targets.

Tolerance: the FP32 kernels' stated bar, relative L2 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


@pytest.mark.parametrize("nt,ns", [(11001, 11363), (11001, 11365), (1001, 125001), (63001, 1999), (257, 500001)])
def test_targets_and_sources(mf, cuda, oracle, nt, ns):
    rng = np.random.default_rng(nt)
    s = rng.random((ns, 3)).astype(np.float32)
    t = (rng.random((nt, 3)) * 1.2 - 0.1).astype(np.float32)
    t[:5] = s[:5]
    m = (rng.normal(size=(ns, 3)) + [0, 0, 2]).astype(np.float32)
    h = float(np.float32(2.0 * ns ** (-1 / 3)))
    idx = np.r_[0:8, nt - 8:nt, rng.choice(nt, 48, replace=False)]
    ds, dt, dm = dev(cuda, s), dev(cuda, t), dev(cuda, m)
    sd, td, md = (v.astype(np.float64) for v in (s, t[idx], m))
    assert rel(mf.direct_field(dt, ds, dm, h).cpu().numpy()[idx], oracle.field(td, sd, md, h)) < TOL
    want = oracle.tensor_sum(td, sd, md, h).reshape(len(idx), 9)
    assert rel(mf.direct_force_tensor(dt, ds, dm, h).cpu().numpy()[idx], want) < TOL


@pytest.mark.parametrize("n", [11180, 11181])
def test_one_set(mf, cuda, oracle, n):
    rng = np.random.default_rng(n)
    s = rng.random((n, 3)).astype(np.float32)
    m = (rng.normal(size=(n, 3)) + [0, 0, 2]).astype(np.float32)
    h = float(np.float32(2.0 * n ** (-1 / 3)))
    idx = np.r_[0:8, n - 8:n, rng.choice(n, 48, replace=False)]
    ds, dm = dev(cuda, s), dev(cuda, m)
    sd, md = s.astype(np.float64), m.astype(np.float64)
    assert rel(mf.direct_field(ds, ds, dm, h).cpu().numpy()[idx], oracle.field(sd[idx], sd, md, h)) < TOL
    T = oracle.tensor_sum(sd[idx], sd, md, h).reshape(-1, 3, 3)
    assert rel(mf.direct_force(ds, dm, h).cpu().numpy()[idx], np.einsum("icr,ic->ir", T, md[idx])) < TOL

"""The FP32 field at smoothing lengths near the ends of FP32's range: h^-5 of the
near form overflows from h = 1e-8 down (point dipoles at ordinary distances)
and is subnormal from h = 1e8 up.

Tolerance: the FP32 kernels' stated bar against the FP64 oracle, relative L2
1e-5; at 1e8 the coefficients themselves are FP32 subnormals, of which a pair
keeps 17 bits or more: the bar is the same.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


def rel(a, b):
    return np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b)


def dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


def cloud(n, scale=1.0):
    rng = np.random.default_rng(n)
    return (rng.random((n, 3)) * scale).astype(np.float32), rng.normal(size=(n, 3)).astype(np.float32)


@pytest.mark.parametrize("h", [1e-7, 1.5e-8, 9e-9, 1e-9, 1e-12])
def test_small_h(mf, cuda, oracle, h):
    p, m = cloud(200)
    h = float(np.float32(h))
    want = oracle.field(p.astype(np.float64), p.astype(np.float64), m, h)
    s = mf.Solver(len(p), h, h, 1e-3, 1.0, (0, 0, 1), None, None, p)
    assert rel(s.apply_field(m), want) < TOL
    s.close()
    assert rel(mf.direct_field(dev(cuda, p), dev(cuda, p), dev(cuda, m), h).cpu().numpy(), want) < TOL


def test_small_h_packed(mf, cuda, oracle):
    p, m = cloud(3000)
    h = float(np.float32(1.5e-8))
    s = mf.Solver(len(p), h, h, 1e-3, 1.0, (0, 0, 1), None, None, p)
    assert rel(s.apply_field(m), oracle.field(p.astype(np.float64), p.astype(np.float64), m, h)) < TOL
    s.close()


@pytest.mark.parametrize("scale", [1e5, 1e7, 1e8])
def test_large_h(mf, cuda, oracle, scale):
    p, m = cloud(200, scale)
    h = float(np.float32(0.4 * scale))
    want = oracle.field(p.astype(np.float64), p.astype(np.float64), m, h)
    assert rel(mf.direct_field(dev(cuda, p), dev(cuda, p), dev(cuda, m), h).cpu().numpy(), want) < TOL

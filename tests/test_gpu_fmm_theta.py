"""The FMM matrix at apertures so small that no box pair is far: everything is
summed near, whatever the radius 1 / theta squared comes to.

Tolerance: only rounding is left, the FP32 kernels' stated bar 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("theta", [1e-2, 1e-3, 1e-9, 1e-10, 1e-300])
@pytest.mark.parametrize("n", [1, 3000])
def test_everything_near(mf, oracle, theta, n):
    rng = np.random.default_rng(n)
    p = rng.random((n, 3)).astype(np.float32)
    t = rng.random((70, 3)).astype(np.float32)
    m = rng.normal(size=(n, 3)).astype(np.float32)
    A = mf.FmmMatrix(p, 0.1, targets=t, order=6, theta=theta)
    want = oracle.field(t.astype(np.float64), p.astype(np.float64), m, float(np.float32(0.1)))
    assert np.linalg.norm(A.field(m) - want) / np.linalg.norm(want) < 1e-5
    want = oracle.tensor_sum(t.astype(np.float64), p.astype(np.float64), m.astype(np.float64), float(np.float32(0.1)))
    got = A.hessian(m)
    assert np.linalg.norm(got - want.reshape(-1, 9)) / np.linalg.norm(want) < 1e-5
    A.close()

"""The FP32 force tensor at distances exactly on the joins of the fitted curves
(r = h, 2h, 3h, 4h), where the curves jump: exact-branch kernel and the
near-field correction at separate targets against the FP64 oracle.

Every distance, its square and r / h are exact in FP32 (h a power of two, the
axes and the (1, 2, 2) directions), so FP32 and FP64 take the same piece.
Tolerance: the FP32 kernels' stated bar, 1e-5, for every target by itself.
"""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


def dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


def on_joins(h):
    axes = [np.array(v, float) * s * q for v in np.eye(3) for s in (1, -1) for q in (1, 2, 3, 4)]
    tilted = [np.array(v, float) * s for v in set(itertools.permutations((1, 2, 2)))
              for s in itertools.product((1, -1), repeat=3)]  # length 3
    return (np.array(axes + tilted) * h).astype(np.float32)


@pytest.mark.parametrize("k", [0, 2, 5])
def test_joins(mf, cuda, oracle, k):
    h = 2.0 ** -k
    t = on_joins(h)
    s = np.zeros((1, 3), np.float32)
    m = np.array([[0.3, -0.5, 1.0]], np.float32)
    want = oracle.tensor_sum(t.astype(np.float64), s.astype(np.float64), m, h).reshape(-1, 9)
    A = mf.FmmMatrix(s, h, targets=t, order=8, theta=0.02)
    for got in (mf.direct_force_tensor(dev(cuda, t), dev(cuda, s), dev(cuda, m), h).cpu().numpy(), A.hessian(m)):
        assert (np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)).max() < TOL
    A.close()

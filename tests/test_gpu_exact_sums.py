"""Rounding of the exact-branch FP32 sums.  Small direct calls take the
exact-branch kernels, large ones the packed ones: the same sums (the targets
repeated until the call is large) must not lose accuracy below the line.

Tolerance: the exact-branch sums' error against FP64 is at most 1.1 times the
packed ones' (their FP32 chains, folded into compensated sums, are no longer;
0.1 for the spread between two sets of roundings).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b)


def dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


@pytest.mark.parametrize("n", [1000, 3001, 9000])
def test_field_and_tensor(mf, cuda, oracle, n):
    import scenes
    sc = scenes.jittered_lattice(n, "sphere", chi=2.0, seed=n)
    m = np.asarray(sc.c * (np.array([0.1, -0.2, 1.0]) + 0.3 * np.random.default_rng(n).normal(size=(n, 3))), np.float32)
    h = float(np.float32(sc.h))
    many = np.tile(sc.pos, (int(np.ceil(1.3e8 / n ** 2)), 1))
    p, q, t = dev(cuda, sc.pos), dev(cuda, m), dev(cuda, many)
    pd = sc.pos.astype(np.float64)
    want = oracle.field(pd, pd, m, h)
    exact, packed = mf.direct_field(p, p, q, h), mf.direct_field(t, p, q, h)[:n]
    assert rel(exact.cpu().numpy(), want) <= 1.1 * rel(packed.cpu().numpy(), want)
    want = oracle.tensor_sum(pd, pd, m.astype(np.float64), h).reshape(-1, 9)
    exact, packed = mf.direct_force_tensor(p, p, q, h), mf.direct_force_tensor(t, p, q, h)[:n]
    assert rel(exact.cpu().numpy(), want) <= 1.1 * rel(packed.cpu().numpy(), want)

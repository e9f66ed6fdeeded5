"""Direct calls whose counts or density are lopsided take the kernel that serves
them: compared with calls of the same kind right beside them.

Bounds: the work of the two sides differs by the stated factor; half as much
again is allowed for launches and noise, three quarters for the dense sets, whose
bounding box is read first (the wrong kernel took 3.4, 1.7, 2 and 5 times).
"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def best(torch, f, n=12):
    for _ in range(3):
        f()
    torch.cuda.synchronize()
    t = []
    for _ in range(n):
        t0 = time.perf_counter()
        f()
        torch.cuda.synchronize()
        t.append(time.perf_counter() - t0)
    return min(t)


def sets(torch, nt, ns):
    g = torch.Generator(device="cuda").manual_seed(nt)
    r = lambda n: torch.rand((n, 3), generator=g, device="cuda")
    return r(nt), r(ns), torch.randn((ns, 3), generator=g, device="cuda")


def test_tensor_of_few_sources(mf, cuda):
    t, s, m = sets(cuda, 1000000, 126)
    whole = best(cuda, lambda: mf.direct_force_tensor(t, s, m, 0.1))
    half = best(cuda, lambda: mf.direct_force_tensor(t[:500000], s, m, 0.1))
    assert whole < 1.5 * 2 * half


def test_field_at_few_targets(mf, cuda):
    t, s, m = sets(cuda, 16, 10000000)
    ten = best(cuda, lambda: mf.direct_field(t[:10], s, m, 0.01))
    all_ = best(cuda, lambda: mf.direct_field(t, s, m, 0.01))
    assert ten < 1.5 * all_


def test_tensor_of_dense_sources(mf, cuda):
    t, s, m = sets(cuda, 12000, 12000)
    whole = best(cuda, lambda: mf.direct_force_tensor(t, s, m, 0.4))
    less = best(cuda, lambda: mf.direct_force_tensor(t[:10000], s[:10000], m[:10000], 0.4))
    assert whole < 1.75 * 1.44 * less


def test_field_of_dense_sources(mf, cuda):
    t, s, m = sets(cuda, 12000, 12000)
    dense = best(cuda, lambda: mf.direct_field(s, s, m, 0.3))
    sparse = best(cuda, lambda: mf.direct_field(s, s, m, 0.02))
    assert dense < 1.75 * sparse

"""The FMM's translation on the multi-indices with z <= 1.

CPU: the index maps, the reduction of the multipoles, the translation over the
reduced indices and the completion of the locals, mirrored here, give the full
multi-index sum (FP64, to rounding).  GPU: field products at every expansion
order against the FP64 oracle.

Tolerances.  CPU: both sides are the same sum in another order, at most ~1e4
FP64 terms: 1e-11.  GPU: the stated bars at P = 6 (1e-4) and from P = 8 on
(1e-5); 2e-5 at P = 7; below, the measured 3e-5 of P = 6 times 3.3 per order
(the convergence at aperture 0.5) with a margin of 10.
"""
import math

import numpy as np
import pytest

LAST = 9


def ncoef(q):
    return 0 if q < 0 else (q + 1) * (q + 2) * (q + 3) // 6


def nharm(q):
    return (q + 1) ** 2 - 1


def hidx(x, y, z):
    return nharm(x + y + z - 1) + (y if z == 0 else x + y + 2 + y)


def dofs(n):
    return 0 if n <= 0 else 1 + 3 * n * (n - 1) // 2


def didx(x, y, z):
    n = x + y + z
    return dofs(n) + (y if z == 0 else n + 1 + y if z == 1 else 2 * n + 1 + y)


def indices(lo, hi):
    return [(n - y - z, y, z) for n in range(lo, hi + 1) for z in range(n + 1) for y in range(n - z + 1)]


def derivatives(d, nmax):
    """gamma! times the Taylor coefficients of 1/|d| (FP64 recurrence)."""
    t = {}
    r2 = float(np.dot(d, d))
    for g in sorted(indices(0, nmax), key=sum):
        n = sum(g)
        if n == 0:
            t[g] = 1 / math.sqrt(r2)
            continue
        acc = 0.0
        for i in range(3):
            b = list(g)
            if g[i] >= 1:
                b[i] -= 1
                acc += (2 * n - 1) * d[i] * t[tuple(b)]
            if g[i] >= 2:
                b[i] -= 1
                acc += (n - 1) * t[tuple(b)]
        t[g] = -acc / (n * r2)
    return {g: v * math.factorial(g[0]) * math.factorial(g[1]) * math.factorial(g[2]) for g, v in t.items()}


def test_index_maps():
    h = [g for g in indices(1, LAST) if g[2] <= 1]
    assert sorted(hidx(*g) for g in h) == list(range(nharm(LAST)))
    d = [g for g in indices(0, LAST + 1) if g[2] <= 2]
    assert sorted(didx(*g) for g in d) == list(range(dofs(LAST + 2)))
    # k -> (x, y, z) as the reduction kernel decodes it
    for g in h:
        k, n = hidx(*g), 1
        while k >= nharm(n):
            n += 1
        w = k - nharm(n - 1)
        z = 0 if w <= n else 1
        y = w if w <= n else w - n - 1
        assert (n - z - y, y, z) == g


@pytest.mark.parametrize("q", range(3, LAST + 1))
def test_reduced_translation_is_the_full_sum(q):
    rng = np.random.default_rng(q)
    m = {a: rng.normal() for a in indices(1, q)}
    dd = derivatives(rng.normal(size=3) + np.array([2.0, -1.0, 1.5]), q + 1)
    red = {}
    for (x, y, z) in (g for g in indices(1, q) if g[2] <= 1):
        v = 0.0
        for j in range((x + y) // 2 + 1):
            for i in range(j + 1):
                a, c = x - 2 * i, y - 2 * (j - i)
                if a >= 0 and c >= 0:
                    v += (-1) ** j * math.comb(j, i) * m[(a, c, z + 2 * j)]
        red[(x, y, z)] = v

    def add(a, b):
        return tuple(u + v for u, v in zip(a, b))

    loc = {b: sum(v * dd[add(a, b)] for a, v in red.items() if sum(a) + sum(b) <= q + 1) for b in red}
    for b in indices(1, q):
        full = sum(v * dd[add(a, b)] for a, v in m.items() if sum(a) + sum(b) <= q + 1)
        j, z = b[2] >> 1, b[2] & 1
        got = (-1) ** j * sum(math.comb(j, i) * loc[(b[0] + 2 * i, b[1] + 2 * (j - i), z)] for i in range(j + 1))
        scale = sum(abs(v * dd[add(a, b)]) for a, v in m.items() if sum(a) + sum(b) <= q + 1)
        assert abs(got - full) <= 1e-11 * max(scale, 1e-300), (b, got, full)


@pytest.mark.gpu
@pytest.mark.parametrize("order,tol", [(4, 3.3e-3), (5, 1e-3), (6, 1e-4), (7, 2e-5), (8, 1e-5), (9, 1e-5)])
def test_field_at_every_order(mf, oracle, order, tol):
    import scenes
    sc = scenes.jittered_lattice(20011, "cylinder", radius=0.3, height=1.0, chi=1.5, seed=order)
    rng = np.random.default_rng(order)
    m = ((np.array([0.0, 0.0, 1.0]) + 0.3 * rng.normal(size=(sc.n, 3))) * sc.volume).astype(np.float32)
    a = mf.FmmMatrix(sc.pos, sc.h, order=order, theta=0.5, leaf_min=12)
    idx = rng.choice(sc.n, 512, replace=False)
    want = oracle.field(sc.pos[idx].astype(np.float64), sc.pos.astype(np.float64), m.astype(np.float64), sc.h)
    got = a.field(m)[idx].astype(np.float64)
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < tol

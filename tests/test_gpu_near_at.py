"""The near-field correction at separate targets (one warp per target) against
the FP64 oracle, where its row lists can go wrong: warp remainders, targets
outside the sources' box and on its faces, targets at sources, grids of few and
of many cells, cells without sources.

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


def sources(kind, ns, rng):
    if kind == "cube":
        return rng.random((ns, 3)).astype(np.float32)
    if kind == "slab":  # a flat grid: few cells along z
        return (rng.random((ns, 3)) * [1.0, 1.0, 0.01]).astype(np.float32)
    # two far clusters: most cells empty, cells widened
    p = rng.random((ns, 3)) * 0.2
    p[ns // 2:, 0] += 40.0
    return p.astype(np.float32)


@pytest.mark.parametrize("kind", ["cube", "slab", "clusters"])
@pytest.mark.parametrize("nt,ns,h", [(1, 900, 0.2), (5, 33, 0.5), (131, 4000, 0.03), (1000, 2999, 0.08)])
def test_field_at_separate_targets(mf, cuda, oracle, kind, nt, ns, h):
    rng = np.random.default_rng(nt + ns)
    s = sources(kind, ns, rng)
    lo, hi = s.min(axis=0), s.max(axis=0)
    t = (lo - 3 * h + rng.random((nt, 3)) * (hi - lo + 6 * h)).astype(np.float32)
    k = max(1, nt // 8)
    t[:k] = s[:k] if ns >= k else t[:k]      # at sources (self term)
    t[-k:] = np.where(rng.random((k, 3)) < 0.5, lo, hi)  # corners and edges of the box
    m = rng.normal(size=(ns, 3)).astype(np.float32)
    got = mf.direct_field(dev(cuda, t), dev(cuda, s), dev(cuda, m), h).cpu().numpy()
    assert rel(got, oracle.field(t, s, m, h)) < TOL

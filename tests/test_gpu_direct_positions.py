"""Which source positions the direct calls take, on both sides of the size where
the packed kernels start: the field and the force refuse sources without a
finite bounding box, and leave the results alone; the tensor takes them all.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INF, NAN = np.inf, np.nan


def dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


def bad_sources(n, kind):
    rng = np.random.default_rng(n)
    s = rng.random((n, 3)).astype(np.float32)
    if kind == "one inf":
        s[7, 1] = INF
    elif kind == "last -inf":
        s[-1, 2] = -INF
    elif kind == "one nan":
        s[7, 1] = NAN
    elif kind == "nan axis":
        s[:, 0] = NAN
    return s, rng.normal(size=(n, 3)).astype(np.float32)


def status(mf, f):
    try:
        f()
        return 0
    except mf.MFError as e:
        return e.status


@pytest.mark.parametrize("n", [33, 300, 12000])
@pytest.mark.parametrize("kind,refused", [("finite", 0), ("one inf", 1), ("last -inf", 1), ("one nan", 0), ("nan axis", 1)])
def test_what_is_taken(mf, cuda, n, kind, refused):
    s, m = bad_sources(n, kind)
    ds, dm = dev(cuda, s), dev(cuda, m)
    dt = dev(cuda, np.random.default_rng(1).random((n + 1, 3)))
    out = cuda.full((n + 1, 3), 5.0, device="cuda")
    st = mf.load().mf_direct_field(mf._dev(dt), n + 1, mf._dev(ds), mf._dev(dm), n, 0.1, mf._dev(out), mf._stream())
    assert st == refused
    assert bool((out == 5.0).all()) == bool(refused)
    assert status(mf, lambda: mf.direct_field(ds, ds, dm, 0.1)) == refused
    assert status(mf, lambda: mf.direct_force(ds, dm, 0.1)) == refused
    assert status(mf, lambda: mf.direct_force_tensor(dt, ds, dm, 0.1)) == 0
    # and the next call is as if nothing had been
    good = dev(cuda, bad_sources(n, "finite")[0])
    assert bool(cuda.isfinite(mf.direct_field(good, good, dm, 0.1)).all())


def test_tensor_of_sources_too_spread_for_cells(mf, cuda, oracle):
    """Two clusters 1e6 apart at h = 1e-3: a cell list would need 1e9 cells a side."""
    rng = np.random.default_rng(3)
    s = rng.random((12000, 3)).astype(np.float32)
    s[::2] += np.float32(1e6)
    m = rng.normal(size=s.shape).astype(np.float32)
    h = float(np.float32(1e-3))
    got = mf.direct_force_tensor(dev(cuda, s), dev(cuda, s), dev(cuda, m), h).cpu().numpy()
    k = np.r_[0:40, 11960:12000]
    sd = s.astype(np.float64)
    want = oracle.tensor_sum(sd[k], sd, m.astype(np.float64), h).reshape(-1, 9)
    assert np.linalg.norm(got[k] - want) / np.linalg.norm(want) < 1e-5

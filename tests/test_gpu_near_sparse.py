"""The packed force correction where cells hold few particles (one warp a cell)
and where they are full (four), on both sides of the line, with clumps and a
coincident pair, against the FP64 oracle.

Tolerance: the FP32 kernels' stated bar, relative L2 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


def rel(a, b):
    return np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b)


def dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


@pytest.mark.parametrize("per", [1, 2, 3, 9])
@pytest.mark.parametrize("ratio", [0.6, 1.2, 1.3, 2.0])
def test_clumps(mf, cuda, oracle, per, ratio):
    """n clumps of `per` particles on a lattice; cells of ratio spacings."""
    rng = np.random.default_rng(per)
    side = int(np.ceil((12500 / per) ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    p = ((g + 0.5 + 0.3 * rng.random((len(g), per, 3))).reshape(-1, 3) / side).astype(np.float32)
    p[1] = p[0]
    m = (rng.normal(size=p.shape) + [0, 0, 2]).astype(np.float32)
    h = float(np.float32(ratio / side))
    k = np.r_[0:32, len(p) - 32:len(p)]
    pd, md = p.astype(np.float64), m.astype(np.float64)
    T = oracle.tensor_sum(pd[k], pd, md, h).reshape(-1, 3, 3)
    got = mf.direct_force(dev(cuda, p), dev(cuda, m), h).cpu().numpy()[k]
    assert rel(got, np.einsum("icr,ic->ir", T, md[k])) < TOL

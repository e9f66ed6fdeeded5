"""GPU test of a batch's read-back (mf_batch_get): what was put in comes out
bit for bit, for scenes of any size in any order, and M = c b holds scene by
scene, so no value is read from a neighbour's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1,), (2, 255, 1, 2049), (33, 4097, 256, 85, 86)])
def test_every_quantity_comes_back(mf, sizes):
    import scenes
    scs = [scenes.jittered_lattice(n, "sphere", radius=0.3, chi=0.5 + 0.4 * k, seed=40 + k, H0=(0.1 * k, 1.0, -0.3))
           for k, n in enumerate(sizes)]
    b = mf.Batch(scs)
    b.solve(50, 1e-6)
    b.eval_force()
    order = list(np.argsort(sizes))
    for k in order + order[::-1]:
        sc = scs[k]
        assert np.array_equal(b.get(k, "positions"), np.asarray(sc.pos, np.float32))
        assert np.array_equal(b.get(k, "Hext"), np.broadcast_to(np.asarray(sc.H0, np.float32), (sc.n, 3)))
        m, f = b.get(k, "M"), b.get(k, "magnetic_bodyforce")
        assert m.shape == f.shape == (sc.n, 3) and np.isfinite(f).all()
        # roundings of 2^-24: volume, chi, c and the product; twice that is allowed
        np.testing.assert_allclose(m, sc.c * b.get(k, "total_B_over_mu0").astype(np.float64), rtol=2.0 ** -21, atol=0)
    b.close()

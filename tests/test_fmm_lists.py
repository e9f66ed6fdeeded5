"""The FMM's interaction lists from whole-number acceptance radii.

CPU: |d|^2 > m accepts exactly the offsets that the two distance tests accept.
GPU: a handle whose particles move through grids of other shapes and box sizes
(lists kept while they still hold, rebuilt when not) gives the field a fresh
handle gives for the same particles, bit for bit, and the force of its own
magnetization to the FP32 bar (1e-5) against direct sums.
"""
import math

import numpy as np
import pytest


def largest_near(theta, s, rnear):
    r12 = math.sqrt(3.0)

    def far(d2):
        r0 = math.sqrt(float(d2))
        return theta * r0 > r12 and (r0 - r12) * s > rnear

    t = max(r12 / theta, r12 + rnear / s)
    d2 = int(t * t)
    while d2 > 0 and far(d2):
        d2 -= 1
    while not far(d2 + 1):
        d2 += 1
    return d2, far


@pytest.mark.parametrize("theta", [0.2, 0.36, 0.44, 0.5, math.sqrt(3.0) / 4, 1.0])
def test_whole_number_acceptance(theta):
    rng = np.random.default_rng(int(theta * 1000))
    for k in range(40):
        s = float(np.float32(10.0 ** rng.uniform(-3, 0)))
        rnear = s * float(10.0 ** rng.uniform(-2, 1)) if k else s * (4.0 - math.sqrt(3.0))  # first: a test on a whole offset
        m, far = largest_near(theta, s, rnear)
        for d2 in range(0, max(200, 2 * m)):
            assert (d2 > m) == far(d2), (theta, s, rnear, d2, m)


@pytest.mark.gpu
def test_moving_particles_keep_or_rebuild_the_lists(mf, cuda):
    rng = np.random.default_rng(1)
    n = 12001
    base = rng.random((n, 3)).astype(np.float32)
    m = rng.normal(size=(n, 3)).astype(np.float32)
    h = 0.02

    def handle(pos):
        s = mf.Solver(n, h, h, 1e-4, 1.0, (0.0, 0.0, 1.0), None, None, pos)
        s.set_option("fmm", mf.FMM_ON)
        return s

    moving = handle(base)
    for scale in ((1, 1, 1), (1.001, 1, 0.999), (1, 1, 2.2), (0.5, 0.5, 0.5), (0.5, 0.5, 0.5001), (1, 1, 1), (3, 0.2, 1)):
        pos = (base * np.asarray(scale, np.float32)).astype(np.float32)
        moving.setTargetpos(pos)
        fresh = handle(pos)
        assert np.array_equal(moving.apply_field(m), fresh.apply_field(m)), scale
        fresh.close()
        moving.solve(0)
        moving.evaluate_fitted_near_foece()
        f = moving.magnetic_bodyforce.astype(np.float64)
        p, q = cuda.from_numpy(pos).cuda(), cuda.from_numpy(moving.M).cuda()
        want = mf.direct_force(p, q, h).cpu().numpy().astype(np.float64)
        assert np.linalg.norm(f - want) < 1e-5 * np.linalg.norm(want), scale
    moving.close()

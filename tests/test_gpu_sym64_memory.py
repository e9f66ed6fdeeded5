"""FP64 handles where the once-per-pair kernels' block sums (0.4 GB at 65,536
particles) cannot be allocated: all pairs, as above 65,536, and the same values.

Values: both kernels sum the same FP64 terms, read back in FP32: 1e-6 of the
largest.  The memory is held by one ordinary allocation of all but 0.25 GB of
what is free.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def product(mf, n):
    rng = np.random.default_rng(n)
    pos = rng.random((n, 3)).astype(np.float32)
    m = rng.normal(size=(n, 3)).astype(np.float32)
    v = 1.0 / n
    s = mf.Solver(n, 2 * v ** (1 / 3), 0.1, v, 0.5, (0, 0, 1), None, None, pos, precision="fp64")
    s.set_option("kernel_timing", 1)
    out = s.apply_field(m)
    k = s.kernel_stats("field")
    s.close()
    return out, k["evals"] < k["pairs"]


def test_no_room_for_the_block_sums(mf, cuda):
    n = 65536
    mf.load().mf_release_scratch()
    cuda.cuda.empty_cache()
    want, once = product(mf, n)
    assert once
    free, _ = cuda.cuda.mem_get_info()
    hold = cuda.empty(free - (250 << 20), dtype=cuda.uint8, device="cuda")
    try:
        got, once = product(mf, n)
    finally:
        del hold
        cuda.cuda.empty_cache()
    assert not once
    assert np.abs(got.astype(float) - want).max() <= 1e-6 * np.abs(want).max()  # FP32 read-back
    assert product(mf, n)[1]


@pytest.mark.parametrize("n,once", [(65536, True), (65537, False)])
def test_limit(mf, cuda, n, once):
    assert product(mf, n)[1] == once

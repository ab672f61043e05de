"""The frame of ordered sums: the caller's, 0 without one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_ordered_fp64_sums_keep_the_callers_frame():
    """K(y, x) a without an origin evaluates the coordinates as they are given: near targets among far ones keep the
    rounding of their own distance (the bound of the exponential's range test), whatever block they are in."""
    from base.kernelFunctions import Kernel
    K = Kernel(name='gauss', sigma=0.5)
    K.pk_dtype = 'float64'
    rng = np.random.default_rng(3)
    r = rng.uniform(0.0, 2.0, size=512)
    far = np.zeros(512, dtype=bool)
    for b in (32, 64, 128):
        for k in range(0, 512, b):
            far[[k, k + (b - 1) // 2, k + b - 1]] = True
    y = np.zeros((512, 3))
    y[:, 1] = np.where(far, 1.0e6 + r, r)
    k = K.applyK(np.zeros((1, 3)), np.ones((1, 3)), firstVar=y)[:, 0]
    t = 0.5 * (r / 0.5) ** 2
    ref = np.exp(-t)
    assert np.all(k[far] == 0)
    assert np.all((np.abs(k - ref) <= (3.5 + 10 * t) * 2.0 ** -53 * ref)[~far])

"""The split symmetric kernels (the warps of a CTA share the targets and divide every source tile) at the edges of their
tiles, row blocks and size ranges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 63, 65, 127, 128, 129, 257, 1280, 1281, 2048, 2049, 3600, 3601, 8192, 8193, 16384, 16385]


@pytest.mark.parametrize('name', ['gauss', 'laplacian'])
@pytest.mark.parametrize('n', SIZES)
def test_fp32_self_sums_against_fp64_ordered(n, name):
    """K a, the second-order steps and the first-order adjoint step in FP32 against the FP64 ordered-pair kernels (a
    distinct target array). Tolerance: the FP32 bound of the other kernel tests, 2e-5 relative on random signs
    (Laplacian 3e-5), 1e-6 of the largest term where a sum of a few points cancels."""
    import torch
    from base import pointEvolution as evol
    from base.kernelFunctions import Kernel
    rng = np.random.default_rng(n)
    X, A, PX, PA = (torch.from_numpy(rng.normal(size=(n, 3))).cuda() for _ in range(4))
    Y = X.clone()
    K, K64 = Kernel(name=name, sigma=0.8, order=3), Kernel(name=name, sigma=0.8, order=3)
    K.pk_dtype, K64.pk_dtype = 'float32', 'float64'
    tol = 2e-5 if name == 'gauss' else 3e-5
    o = [0.1, 0.2, -0.1]

    def close(a, b, size):
        return float((a - b).norm()) <= tol * float(b.norm()) + 1e-6 * size * n ** 0.5

    ka = K64.applyK(X, A, firstVar=Y)
    assert close(K.applyK(X, A), ka, 3.0)
    xt, at = evol.shoot_second_order(X, A, K, 1.0, origin=o)
    assert close(xt[1] - X, ka, 3.0)
    assert close(at[1] - A, -K64.applyDiffKT(X, A, A, firstVar=Y), 10.0)
    pxt, pat, _ = evol.second_order_adjoint(xt, at, PX, PA, K, 1.0, origin=o, with_da0=False)
    zpx = K64.applyDiffKT(X, PX, A, firstVar=Y, sym=True) - K64.applyDDiffK11and12(X, A, A, PA)
    zpa = K64.applyK(X, PX, firstVar=Y) - K64.applyDiffK1and2(X, PA, A)
    assert close(pxt[0] - PX, zpx, 30.0)
    assert close(pat[0] - PA, zpa, 30.0)
    f1, f0 = evol.first_order_gradient(torch.stack([X, X]), A[None].contiguous(), PX, K, 0.5, euclidean=True, origin=o)
    assert close(f1[0] - PX, K64.applyDiffKT(X, PX, A, firstVar=Y, regweight=0.5, lddmm=True), 30.0)
    assert close(f0[0], K64.applyK(X, A - PX, firstVar=Y), 10.0)

"""The FP64 self-sums (each unordered pair once) and their exponential, at the sizes and arguments where they change."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [1, 2, 63, 64, 65, 129, 255, 257, 1000, 2047, 2048, 2049, 2305, 4100])
@pytest.mark.parametrize('name', ['gauss', 'laplacian'])
def test_fp64_self_sums_at_block_edges(n, name):
    """FP64 self-sums (K a and the two second-order steps) evaluate each unordered pair once, in 64 x 2 launch shape up
    to 2,048 points and wider ones above; sizes at the edges of tiles, row blocks and the shapes, against the oracle.
    Tolerance: the sums have up to 4,100 terms of FP64 rounding 2^-53 with random signs, 1e-13 relative."""
    import torch
    from base import pointEvolution as evol
    from base.kernelFunctions import Kernel
    rng = np.random.default_rng(n)
    x, a, px, pa = (rng.normal(size=(n, 3)) for _ in range(4))
    K = Kernel(name=name, sigma=0.6, order=3)
    K.pk_dtype = 'float64'
    ref = O.apply_k(x, x, a, 0.6) if name == 'gauss' else O.laplacian.apply_k(x, x, a, 0.6, 3)
    assert rel_err(K.applyK(x, a), ref) < 1e-13
    X, A, PX, PA = (torch.from_numpy(v).cuda() for v in (x, a, px, pa))
    Y = X.clone()                                                # a distinct array: the ordered-pair kernels
    if name == 'gauss':
        zpx, zpa = O.second_order_adjoint_step_rows(x, a, px, pa, np.arange(n), 0.6)
    else:
        zpx = (K.applyDiffKT(X, PX, A, firstVar=Y, sym=True) - K.applyDDiffK11and12(X, A, A, PA)).cpu().numpy()
        zpa = (K.applyK(X, PX, firstVar=Y) - K.applyDiffK1and2(X, PA, A)).cpu().numpy()
    # the states after one step of size 1 (state plus sum: the difference of two states would lose the sum's digits)
    xt, at = evol.shoot_second_order(X, A, K, 1.0, origin=[0., 0., 0.])
    za = -K.applyDiffKT(X, A, A, firstVar=Y)
    assert rel_err(xt[1].cpu().numpy(), x + ref) < 1e-13
    assert rel_err(at[1].cpu().numpy(), a + za.cpu().numpy()) < 1e-12
    pxt, pat, _ = evol.second_order_adjoint(xt, at, PX, PA, K, 1.0, origin=[0., 0., 0.], with_da0=False)
    assert rel_err(pxt[0].cpu().numpy(), px + zpx) < 1e-12
    assert rel_err(pat[0].cpu().numpy(), pa + zpa) < 1e-12


def test_fp64_exponential_range():
    """The FP64 kernels' exponential against numpy over its whole range: K(y, x) of single pairs at distances from 0 to
    60 widths (values down to the smallest normal number, zeros below it), infinities and NaN. Error: the scaled
    squared distance carries ten roundings at most (two of the scale, one per product, each twice in the square, those
    of numpy's argument beside them), an error of e t each, and the exponential and the reference 3.5 units."""
    import torch
    from base.kernelFunctions import Kernel
    K = Kernel(name='gauss', sigma=0.5)
    K.pk_dtype = 'float64'
    r = np.concatenate([np.linspace(0, 60, 4001), [0.5 ** k for k in range(1, 60)], [38.6, 38.7, 1e6, 1e160]]) * 0.5
    y = np.zeros((r.size, 3))
    y[:, 1] = r
    k = K.applyK(np.zeros((1, 3)), np.ones((1, 3)), firstVar=y)[:, 0]
    with np.errstate(over='ignore'):
        t = 0.5 * (r / 0.5) ** 2
    with np.errstate(over='ignore', under='ignore'):
        ref = np.exp(-t)
    normal = ref >= 2.0 ** -1021
    assert np.all(np.abs(k - ref)[normal] <= (3.5 + 10 * t[normal]) * 2.0 ** -53 * ref[normal])
    assert np.all((k[~normal] >= 0) & (k[~normal] <= 2.0 ** -1020)) and np.all(k[t > 750] == 0)
    bad = K.applyK(np.array([[0., 0., 0.], [1., 0., 0.]]), np.ones((2, 3)), firstVar=np.array([[np.nan, 0., 0.],
                                                                                              [np.inf, 0., 0.]]))
    assert np.all(np.isnan(bad[0])) and np.all(bad[1] == 0)

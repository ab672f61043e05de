"""The symmetric kernels of whole tiles (two sources to a packed operand): the edges of their chunks, tiles and row
blocks, in the range where they are used, and both sides of the rule between them and the split shapes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 16,385 = 128 * 128 + 1; rows of 512, 768, 1,024 and 1,280 points end at 16,384, 16,896 and 17,920; 64-source chunks at
# 16,448; 10,242 points fill the resident CTAs of whole tiles, 13,000 do not
SIZES = [10242, 13000, 16385, 16447, 16448, 16449, 16895, 16896, 16897, 17920, 17921]


@pytest.mark.parametrize('name,order', [('gauss', None), ('laplacian', 3), ('laplacian', 4)])
@pytest.mark.parametrize('n', SIZES)
def test_whole_tiles_against_fp64(n, name, order):
    """Against the FP64 kernels; 2e-5 relative, the bound of the FP32 kernel tests (Laplacian 3e-5)."""
    import torch
    from base import pointEvolution as evol
    from base.kernelFunctions import Kernel
    rng = np.random.default_rng(n)
    X, A, PX, PA = (torch.from_numpy(rng.normal(size=(n, 3))).cuda() for _ in range(4))
    tol = 2e-5 if name == 'gauss' else 3e-5
    out = {}
    for dtype in ('float32', 'float64'):
        K = Kernel(name=name, sigma=0.8) if order is None else Kernel(name=name, sigma=0.8, order=order)
        K.pk_dtype = dtype
        o = [0.1, 0.2, -0.1]
        xt, at = evol.shoot_second_order(X, A, K, 1.0, origin=o)
        pxt, pat, _ = evol.second_order_adjoint(torch.stack([X, X]), torch.stack([A, A]), PX, PA, K, 1.0, origin=o,
                                                with_da0=False)
        f1, f0 = evol.first_order_gradient(torch.stack([X, X]), A[None].contiguous(), PX, K, 0.5, euclidean=True,
                                           origin=o)
        out[dtype] = [K.applyK(X, A), xt[1] - X, at[1] - A, pxt[0] - PX, pat[0] - PA, f1[0] - PX, f0[0]]
    for k, (a, b) in enumerate(zip(out['float32'], out['float64'])):
        assert float((a - b).norm()) <= tol * float(b.norm()), k
        # the last points, where a block, a tile and a chunk end
        assert float((a[-70:] - b[-70:]).norm()) <= 5 * tol * float(b[-70:].norm()), k

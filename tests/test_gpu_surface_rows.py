"""Vertex arrays and weights that do not match the faces of a data term: rows beyond the last referenced vertex are
isolated points, too few are an error on the host (the kernels index by the faces)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _term(**kw):
    from base.kernelFunctions import Kernel
    from base.surfaceDistances import SurfaceDataTerm
    from base.syntheticShapes import icosphere
    v, f = icosphere(2)
    K = Kernel(name='gauss', sigma=kw.pop('sigma', 0.4))
    return SurfaceDataTerm(f, v * [1.1, 1.0, 0.9], f, K, **kw), torch.as_tensor(v, device='cuda')


@pytest.mark.parametrize('sigma', [0.4, [0.3, 0.6]])
@pytest.mark.parametrize('extra', [1, 500])
def test_isolated_points_after_the_last_vertex(extra, sigma):
    """Without `nv` the term knows the vertices of its faces only: further rows have a zero gradient."""
    term, x = _term(sigma=sigma)
    n = x.shape[0]
    more = torch.cat([x, torch.randn(extra, 3, dtype=x.dtype, device=x.device)])
    assert torch.equal(term.energy(more), term.energy(x))
    g, gw = term.gradient(more, with_weights=True)
    r, rw = term.gradient(x, with_weights=True)
    assert torch.equal(g[:n], r) and torch.equal(gw[:n], rw)
    assert g.shape == more.shape and not g[n:].any() and not gw[n:].any()
    known, _ = _term(sigma=sigma, nv=n + extra)
    assert torch.equal(known.gradient(more), g)
    assert torch.equal(known.gradient(x), r)          # `nv` may count points that a shorter array does not have


def test_too_few_rows_or_weights_are_refused():
    term, x = _term()
    for call in (term.energy, term.gradient):
        with pytest.raises(ValueError):
            call(x[:-1])
    n = x.shape[0]
    with pytest.raises(ValueError):
        _term(weights=np.ones(n - 1))
    with pytest.raises(ValueError):
        _term(target_weights=np.ones(n - 1))
    _term(weights=np.ones(n), target_weights=np.ones(n))

"""Entry points of the network's training step that the model itself does not call in this form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('form', ['generator', 'tuple', 'map', 'longer'])
def test_adam_takes_any_iterable_of_gradients(form):
    """The update reads the gradients in turn, as many as there are tensors: the same bits as from a list."""
    import torch
    from base.learnedProposal import MomentumProposal
    a, b = MomentumProposal(seed=1), MomentumProposal(seed=1)
    g = torch.Generator(device='cuda').manual_seed(2)
    grads = [torch.randn(p.shape, generator=g, device='cuda') for p in a.W + a.b]
    a.adam(grads, lr=1e-2)
    b.adam({'generator': (v for v in grads), 'tuple': tuple(grads), 'map': map(torch.clone, grads),
            'longer': grads + grads}[form], lr=1e-2)
    assert all(torch.equal(p, q) for p, q in zip(a.W + a.b + a.Wb, b.W + b.b + b.Wb))



@pytest.mark.parametrize('M,N', [(1, 1), (64, 64), (255, 33), (256, 128), (257, 64), (5000, 100)])
def test_bf16_column_sums(M, N):
    """lddmm_bf16_colsum with its two-pass scratch and without, against float64. Tolerance: FP32 sums of M terms in
    chains of at most M / 8 + 8 additions, 2^-24 of the sum of magnitudes each."""
    import torch
    import base._native as nat
    g = torch.Generator(device='cuda').manual_seed(M + N)
    dy = torch.randn((M, N), generator=g, device='cuda').to(torch.bfloat16)
    ref, mag = dy.double().sum(0), dy.double().abs().sum(0)
    tol = (M / 8 + 8) * 2.0 ** -24 * mag + 1e-30
    ws = torch.empty(((M + 255) // 256) * N, dtype=torch.float32, device='cuda')
    for w in (ws, None):
        db = torch.full((N,), np.nan, dtype=torch.float32, device='cuda')
        nat.check(nat.lib().lddmm_bf16_colsum(nat.ptr(dy), M, N, nat.ptr(db), nat.ptr(w),
                                              0 if w is None else w.numel() * 4, nat.stream_ptr()), 'colsum')
        assert bool(((db.double() - ref).abs() <= tol).all())

"""Entry points of the network's training step that the model itself does not call in this form."""
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


"""The network's training step in one library call: gradients at row counts around the splits of the weight gradients,
against the float64 restatement, and the fused Adam update."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('M,valid', [(64, 64), (128, 100), (512, 512), (1024, 1000), (1088, 1), (33024, 33000)])
def test_gradients_at_split_edges(M, valid):
    """Tolerance: 1e-2 against the oracle that rounds to bf16 at the same points (a sum of rounded terms may differ in
    the last bit of a bf16 activation)."""
    import torch
    from oracle.learned import mlp_loss_and_grads_bf16
    from base.learnedProposal import MomentumProposal, IN_DIM, N_FEATURES, N_OUT
    model = MomentumProposal(seed=5)
    g = torch.Generator(device='cuda').manual_seed(M)
    F = torch.zeros((M, IN_DIM), device='cuda')
    F[:valid, :N_FEATURES] = torch.randn((valid, N_FEATURES), generator=g, device='cuda')
    F = F.to(torch.bfloat16)
    T = torch.randn((M, N_OUT), generator=g, device='cuda')
    for b in model.b:
        b.normal_(0.0, 0.1, generator=g)
    loss, grads = model.gradients(F, T, valid, weight=1.0 / valid)
    # rows past `valid` carry no loss: the oracle sees the valid ones
    ref_loss, _, ref = mlp_loss_and_grads_bf16(F[:valid].float(), [w.float() for w in model.Wb], model.b, T[:valid],
                                               N_OUT, 1.0 / valid)
    assert loss.shape == () and abs(float(loss) - float(ref_loss)) < 1e-2 * float(ref_loss)
    for k, (a, r) in enumerate(zip(grads, ref)):
        assert a.dtype == torch.float32 and a.is_contiguous()
        if float(r.norm()) == 0.0:
            assert float(a.norm()) == 0.0
        else:
            assert rel_err(a.cpu().double().numpy(), r.numpy()) < 1e-2, k
    again = model.gradients(F, T, valid, weight=1.0 / valid)
    assert torch.equal(again[0], loss) and all(torch.equal(a, b) for a, b in zip(again[1], grads))
    acts = model.forward(F, keep=True)
    assert torch.equal(acts[0], model.forward(F)) and [a.shape[1] for a in acts[1]] == [64, 128, 128, 128]


def test_adam_steps_match_the_formula():
    import torch
    from base.learnedProposal import MomentumProposal
    model = MomentumProposal(seed=1)
    g = torch.Generator(device='cuda').manual_seed(2)
    params = model.W + model.b
    ref = [(p.double().clone(), torch.zeros_like(p, dtype=torch.float64), torch.zeros_like(p, dtype=torch.float64))
           for p in params]
    for t in range(1, 4):
        grads = [torch.randn(p.shape, generator=g, device='cuda') for p in params]
        model.adam(grads, lr=1e-2, weight_decay=1e-3)
        for k, gr in enumerate(grads):
            p, m, v = ref[k]
            gi = gr.double() + 1e-3 * p
            m = 0.9 * m + 0.1 * gi
            v = 0.999 * v + 0.001 * gi * gi
            p = p - 1e-2 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
            ref[k] = (p, m, v)
    for p, (r, _, _) in zip(params, ref):
        assert np.allclose(p.cpu().numpy(), r.cpu().numpy(), rtol=2e-5, atol=2e-6)
    for wb, w in zip(model.Wb, model.W):
        assert torch.equal(wb, w.to(torch.bfloat16))


@pytest.mark.parametrize('offset', [0, 2, 4, 6])
@pytest.mark.parametrize('epi', [2, 3, 4])
def test_bf16_outputs_and_mask_aligned_to_a_column_pair(offset, epi):
    """C and the mask of a BF16 epilogue at any 4-byte boundary: the same bits as at a 16-byte one, and nothing beside
    them is written."""
    import torch
    import base._native as nat
    M, N, K = 128, 128, 64
    g = torch.Generator(device='cuda').manual_seed(3)
    A, B = (torch.randn(s, generator=g, device='cuda').to(torch.bfloat16) for s in ((M, K), (K, N)))
    bias, mask = torch.randn(N, generator=g, device='cuda'), torch.randn((M, N), generator=g, device='cuda')
    outs = []
    for off in (0, offset):
        buf = torch.full((M * N + 16,), 7.0, dtype=torch.bfloat16, device='cuda')
        mb = torch.zeros(M * N + 16, dtype=torch.bfloat16, device='cuda')
        C, mk = buf[off:off + M * N], mb[off:off + M * N]
        mk.copy_(mask.reshape(-1))
        nat.check(nat.lib().lddmm_bf16_gemm(0, 0, epi, M, N, K, nat.ptr(A), nat.ptr(B), nat.ptr(bias), nat.ptr(mk),
                                            nat.ptr(C), 1, None, 0, nat.stream_ptr()), 'gemm')
        assert torch.all(buf[:off] == 7.0) and torch.all(buf[off + M * N:] == 7.0)
        outs.append(C.clone())
    assert torch.equal(*outs)


def test_adam_with_fewer_gradients_than_tensors():
    """The weights alone: the tensors without a gradient stay as they are."""
    import torch
    from base.learnedProposal import MomentumProposal
    model = MomentumProposal(seed=1)
    before = [p.clone() for p in model.W + model.b]
    model.adam([torch.ones_like(w) for w in model.W], lr=1e-2)
    assert all(not torch.equal(p, q) for p, q in zip(model.W, before))
    assert all(torch.equal(p, q) for p, q in zip(model.b, before[len(model.W):]))
    model.adam([])
    assert model.step == 2

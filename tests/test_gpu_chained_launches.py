"""Chained (programmatic dependent) launches beside other streams: a captured graph that forks and joins, and kernels of
the framework between copies and kernels of torch, give the bits of the serial calls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [700, 9000])
def test_fork_and_join_in_a_captured_graph(n):
    import torch
    from base import _native as nat
    lib, p = nat.lib(), nat.ptr
    rng = np.random.default_rng(n)
    X, A, B = (torch.from_numpy(rng.normal(size=(n, 3)) / 10).cuda() for _ in range(3))
    out = [torch.empty_like(X) for _ in range(5)]
    nbytes = lib.lddmm_workspace_bytes(n, n, nat.FP32C)
    ws = [torch.empty(nbytes, dtype=torch.uint8, device='cuda') for _ in range(2)]

    def k(dst, x, a, w):
        nat.check(lib.lddmm_apply_k(p(x), n, p(x), p(a), n, 0.5, nat.KERNEL_GAUSS, None, p(dst), nat.FP32C, p(w), nbytes,
                                    nat.stream_ptr()), 'apply_k')

    side = torch.cuda.Stream()

    def step():
        k(out[0], X, A, ws[0])
        side.wait_stream(torch.cuda.current_stream())           # the side stream starts from a chained kernel
        with torch.cuda.stream(side):
            k(out[1], X, out[0], ws[1])
            k(out[2], X, out[1], ws[1])
        out[3].copy_(out[0])
        out[3].add_(B)
        k(out[3], X, out[3].clone(), ws[0])
        torch.cuda.current_stream().wait_stream(side)           # and a chained kernel has two predecessors
        k(out[4], X, out[2], ws[0])
        out[4].add_(out[3])

    main = torch.cuda.Stream()
    main.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(main):
        step()
    main.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        step()
    for _ in range(3):
        A.copy_(torch.from_numpy(rng.normal(size=(n, 3)) / 10))
        g.replay()
        torch.cuda.synchronize()
        got = [o.clone() for o in out]
        ref = []
        for x, a in ((X, A), (X, None), (X, None)):             # serially, each call on its own
            r = torch.empty_like(X)
            k(r, x, a if a is not None else ref[-1], ws[0])
            torch.cuda.synchronize()
            ref.append(r)
        r3 = torch.empty_like(X)
        k(r3, X, ref[0] + B, ws[0])
        r4 = torch.empty_like(X)
        k(r4, X, ref[2], ws[0])
        torch.cuda.synchronize()
        for a, b in zip(got, ref + [r3, r4 + r3]):
            assert torch.equal(a, b)
    del g

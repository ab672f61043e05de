"""The scratch sizes that the library reports hold every launch they are reported for. Host part: relations between the
reported sizes (without a device the plans are those of 148 SMs and the library's default residency). GPU part: calls
with a workspace of exactly the reported size."""
import numpy as np
import pytest


def _lib():
    from base import _native as nat
    return nat.load_library()


def _faces(nf):
    """A triangulated height field of at least nf faces, cut to nf: (vertices, faces)."""
    k = int(np.ceil(np.sqrt(nf / 2))) + 1
    u, v = np.meshgrid(np.linspace(0, 1, k), np.linspace(0, 1, k), indexing='ij')
    x = np.stack([u, v, 0.1 * np.sin(5 * u) * np.cos(4 * v)], axis=-1).reshape(-1, 3)
    i = (np.arange(k - 1)[:, None] * k + np.arange(k - 1)[None]).reshape(-1)
    f = np.stack([np.stack([i, i + k, i + 1], -1), np.stack([i + 1, i + k, i + k + 1], -1)], 1).reshape(-1, 3)
    return np.ascontiguousarray(x), np.ascontiguousarray(f[:nf], dtype=np.int64)


@pytest.mark.parametrize('precision', [0, 1], ids=['fp32c', 'fp64'])
def test_surface_scratch_covers_the_norm_alone(precision):
    """The norm of the target alone is the call with no deformed face, in the scratch of (nf, nf1): equal and unequal
    face counts from one face to the level-6 sphere."""
    size = _lib().lddmm_surface_workspace_bytes
    bad = [(nf, nf1) for nf1 in list(range(1, 42000, 131)) + [20480, 40960, 81920]
           for nf in {nf1, nf1 - 1, nf1 + 1, nf1 // 2, 2 * nf1} if size(nf, nf1, precision) < size(0, nf1, precision)]
    assert not bad, bad[:10]


@pytest.mark.gpu
@pytest.mark.parametrize('precision,nf', [(0, 1), (0, 10496), (0, 12800), (0, 14720), (0, 16500), (0, 20480),
                                          (0, 40960), (1, 1), (1, 6976), (1, 7232)])
def test_surface_calls_in_exactly_the_reported_scratch(precision, nf):
    """Energy, energy with the norm, norm alone and gradient of surfaces of equal face counts, every kind, in exactly the
    reported bytes: accepted, and the same bits as in a larger workspace."""
    import torch
    from base import _native as nat
    lib = nat.lib()
    x, f = _faces(nf)
    X = torch.from_numpy(x).cuda()
    X1 = X + 0.01 * torch.sin(7 * X)
    F = torch.from_numpy(f).cuda()
    nv = x.shape[0]
    from base.surfaceDistances import vertex_face_table
    off, items = vertex_face_table(f, nv)
    o = nat.origin_arg(nat.centroid(X1))
    exact = lib.lddmm_surface_workspace_bytes(nf, nf, precision)
    p = nat.ptr

    def calls(nbytes, kind):
        W = torch.empty(nbytes, dtype=torch.uint8, device='cuda')
        res = []
        for xd, n, with_norm in ((X, nf, 0), (X, nf, 1), (None, 0, 1)):
            e = torch.zeros(2, dtype=torch.float64, device='cuda')
            rc = lib.lddmm_surface_energy(kind, p(xd), nv if n else 0, p(F) if n else None, n, None, p(X1), nv, p(F), nf,
                                          None, 0.1, o, with_norm, p(e), precision, p(W), nbytes, nat.stream_ptr())
            assert rc == 0, (kind, n, with_norm, lib.lddmm_status_string(rc))
            res.append(e)
        g = torch.empty((nv, 3), dtype=torch.float64, device='cuda')
        rc = lib.lddmm_surface_gradient(kind, p(X), nv, p(F), nf, None, p(off), p(items), p(X1), nv, p(F), nf, None, 0.1,
                                        o, p(g), None, precision, p(W), nbytes, nat.stream_ptr())
        assert rc == 0, (kind, lib.lddmm_status_string(rc))
        return res + [g]

    for kind in (nat.DATA_VARIFOLD, nat.DATA_CURRENT, nat.DATA_MEASURE):
        for a, b in zip(calls(exact, kind), calls(2 * exact, kind)):
            assert torch.equal(a, b) and bool(torch.isfinite(a).all()), kind

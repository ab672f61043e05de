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


@pytest.mark.parametrize('precision', [0, 1], ids=['fp32c', 'fp64'])
def test_workspace_bytes_never_falls_with_the_problem(precision):
    """A workspace for n_max targets and m_max sources serves every smaller problem, so its size may not fall as either
    grows (through the ranges where the launch shapes alternate, and past the largest FP64 set of the symmetric kernels)."""
    size = _lib().lddmm_workspace_bytes
    ns = list(range(0, 30000, 61)) + [40962, 100000, 151296, 151297, 163842, 400000]
    for other in (None, 1, 3000, 40962):
        for swap in (False, True):
            got = [size(*((other if other is not None else n, n) if swap else
                          (n, other if other is not None else n)), precision) for n in ns]
            assert got == sorted(got), (other, swap)


def test_ordered_sums_reserve_no_pair_partials():
    """Scratch that grows with the square of the set is asked for by self-sums and shooting steps alone: ordered sums of
    any size take tens of bytes per target, a wide sum of few sources in particular; and a call's own size is never above
    that of the workspace that serves it."""
    lib = _lib()
    call, upto = lib.lddmm_call_workspace_bytes, lib.lddmm_workspace_bytes
    assert upto(200000, 100, 1) < 200 << 20 and upto(100, 200000, 0) < 200 << 20
    for precision in (0, 1):
        for n in (1, 700, 1281, 4097, 8704, 10368, 13000, 40962, 150000, 200000):
            # 12 sums of 8 bytes in at most (resident CTAs x block) / n + 2 slots
            assert call(n, n, 0, precision) <= 96 * (2 * n + 148 * 8 * 1024) + 4096
            assert call(n, 100, 0, precision) <= call(n, n, 0, precision)
            assert call(n, n, 0, precision) <= call(n, n, 1, precision) <= upto(n, n, precision)
            assert call(n, 100, 0, precision) <= upto(n, 100, precision)
    assert call(300000, 300000, 1, 1) < 200 << 20          # above the symmetric FP64 kernels' bounds
    assert call(10, 11, 1, 0) == 0 and call(10, 10, 0, 7) == 0


# --- the plans of csrc/lddmm_common.cuh and csrc/pairs_sym.cuh, restated
def _tri(j):
    return j * (j - 1) // 2


def _row_off(i, TT, TPB, B):
    if B >= TPB:
        return i * TT - (B // TPB) * _tri(i)
    share = TPB // B
    q, r = divmod(i, share)
    return i * TT - (share * _tri(q) + q * r)


def _cta_of(u, W, C):
    return ((u + 1) * C - 1) // W


def _max_slots(length, W, C):
    return -(-(length - 1) * C // W) + 1


def _sym_rows(n, TPB, B, wave):
    """(slots, units, CTAs, tiles, row blocks) of make_sym_plan."""
    nblk, TT = -(-n // B), -(-n // TPB)
    U = _row_off(nblk, TT, TPB, B)
    C = U if 2 * U < 3 * wave else wave
    return _max_slots(TT, U, C), U, C, TT, nblk


def _sym_upto(lo, hi, TPB, B, wave):
    """Slots times points of sym_plan_upto."""
    points = 2 * wave * B + 2 * hi
    if 2 * _sym_rows(lo + 1, TPB, B, wave)[1] < 3 * wave:
        points = max(points, 3 * wave * B)
    return min(points, -(-hi // TPB) * hi)


SHAPES = [(128, 32), (128, 64), (128, 128), (128, 256), (128, 512), (128, 768), (128, 1024), (64, 256), (128, 256)]


@pytest.mark.parametrize('TPB,B', SHAPES)
def test_slots_of_a_symmetric_plan(TPB, B):
    """The slots reserved are those of the longest row, or one more; and the bound over a range of n holds each n's."""
    for wave in (3, 148, 296, 444, 740, 1184):
        ns = sorted(set(range(1, 4000, 173)) | {B - 1, B, B + 1, 8193, 10368, 16384, 20001, 40962})
        need = {}
        for n in ns:
            S, U, C, TT, nblk = _sym_rows(n, TPB, B, wave)
            real = max(_cta_of(_row_off(i + 1, TT, TPB, B) - 1, U, C) - _cta_of(_row_off(i, TT, TPB, B), U, C) + 1
                       for i in range(nblk))
            assert real <= S <= real + 1, (n, wave)
            need[n] = S * n
        for lo in (0, 1408, 8192, 16384):
            for hi in ns:
                inside = [need[n] for n in ns if lo < n <= hi]
                assert not inside or max(inside) <= _sym_upto(lo, hi, TPB, B, wave), (lo, hi, wave)


@pytest.mark.parametrize('TPB,B', [(128, 128), (128, 256), (128, 512), (128, 1024), (128, 64)])
def test_slots_of_an_ordered_plan(TPB, B):
    """Ordered sums and the triangles of the energies: the slots hold the longest row, and slots times targets of a
    smaller ordered problem stay under the bound of the larger one."""
    for wave in (5, 148, 444, 1184):
        need = {}
        ns = [1, 100, B, B + 1, 3000, 13000, 40962, 226301, 262144]
        ts = [1, 2, 3, 24, 100, 161, 321, 7813]
        for n in ns:
            for tiles in ts:
                gx = -(-n // B)
                W = gx * tiles
                C = min(W, wave)
                S = _max_slots(tiles, W, C)
                real = max(_cta_of((i + 1) * tiles - 1, W, C) - _cta_of(i * tiles, W, C) + 1 for i in range(gx))
                assert real <= S <= real + 1
                need[n, tiles] = S * n
                self_tiles = -(-n // TPB)                        # an energy: the self part is a triangle
                W = _row_off(gx, self_tiles + tiles, TPB, B)
                C = min(W, wave)
                off = [_row_off(i, self_tiles + tiles, TPB, B) for i in range(gx + 1)]
                real = max(_cta_of(off[i + 1] - 1, W, C) - _cta_of(off[i], W, C) + 1 for i in range(gx))
                assert real <= _max_slots(self_tiles + tiles, W, C)
        for n in ns:
            for tiles in ts:
                bound = min(n * tiles, wave * B + 2 * n)
                assert max(v for (k, t), v in need.items() if k <= n and t <= tiles) <= bound


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


@pytest.mark.gpu
@pytest.mark.parametrize('precision', [0, 1], ids=['fp32c', 'fp64'])
@pytest.mark.parametrize('kernel', [0, 19, 20], ids=['gauss', 'laplacian3', 'laplacian4'])
def test_smaller_sets_in_the_scratch_of_the_largest(precision, kernel):
    """Self-sums, shooting steps and ordered sums of every size up to n_max in exactly the bytes reported for n_max,
    through the ranges where the launch shapes change."""
    import torch
    from base import _native as nat
    lib = nat.lib()
    rng = np.random.default_rng(kernel)
    n_max = 20000 if precision == 0 else 9000
    X = torch.from_numpy(rng.normal(size=(n_max, 3))).cuda()
    A = torch.from_numpy(rng.normal(size=(n_max, 3)) / n_max).cuda()
    out = [torch.empty((2 * n_max, 3), dtype=torch.float64, device='cuda') for _ in range(2)]
    e = torch.zeros(1, dtype=torch.float64, device='cuda')
    p = nat.ptr
    for top in (n_max, n_max // 2):
        nbytes = lib.lddmm_workspace_bytes(top, top, precision)
        W = torch.empty(nbytes, dtype=torch.uint8, device='cuda')
        end = (precision, p(W), nbytes, nat.stream_ptr())
        ns = {1, 700, 1280, 1281, 1408, 1409, 2304, 2305, 3601, 4097, 4352, 5400, 6500, 7232, 8192, 8445, 8704, 9216, 9984,
              10363, 10368, 10496, 13000, 15000, 16384, 16385, top}
        for n in sorted(k for k in ns if k <= top):
            rcs = {
                'apply_k': lib.lddmm_apply_k(p(X), n, p(X), p(A), n, 0.5, kernel, None, p(out[0]), *end),
                'ordered': lib.lddmm_apply_k(p(A), n, p(X), p(A), n, 0.5, kernel, None, p(out[0]), *end),
                'diff_kt': lib.lddmm_apply_diff_kt(p(X), n, p(X), p(A), p(A), n, 0.5, kernel, 0, 1.0, None, p(out[0]),
                                                   *end),
                'forward': lib.lddmm_second_order_step(p(X), p(A), n, 0.5, kernel, 0.1, None, p(out[0]), p(out[1]), *end),
                'adjoint': lib.lddmm_second_order_adjoint_step(p(X), p(A), p(A), p(A), n, 0.5, kernel, 0.1, None,
                                                               p(out[0]), p(out[1]), *end),
                'rows': lib.lddmm_second_order_adjoint_step_rows(p(X), p(A), p(A), p(A), n, 0, (n + 1) // 2, 0.5, kernel,
                                                                 0.1, None, p(out[0]), p(out[1]), *end),
                'first-order': lib.lddmm_first_order_gradient(p(X), p(A), n, 1, 0.5, kernel, 1.0, p(A), 1, None,
                                                              p(out[0]), p(out[1]), *end),
                'energy': lib.lddmm_first_order_shoot(p(X), p(A), n, 1, 0.5, kernel, 1.0, None, p(out[0]), p(e), *end),
            }
            assert not any(rcs.values()), (top, n, rcs)
    torch.cuda.synchronize()
    assert bool(torch.isfinite(out[0][:n_max // 2]).all())


@pytest.mark.gpu
def test_ordered_fp64_sums_do_not_grow_the_workspace(monkeypatch):
    """K(y, x) a and a derivative operator in FP64, and a self-sum after them in the same buffer."""
    import torch
    from base import _native as nat
    from base.kernelFunctions import Kernel
    monkeypatch.setattr(nat, 'WORKSPACE', nat.Workspace())
    K = Kernel(name='gauss', sigma=0.5)
    K.pk_dtype = 'float64'
    rng = np.random.default_rng(0)
    X = torch.from_numpy(rng.normal(size=(60000, 3))).cuda()
    Y = X + 0.01
    K.applyK(X[:100].contiguous(), X[:100].contiguous(), firstVar=Y)
    K.applyK(X[:3000].contiguous(), X[:3000].contiguous(), firstVar=Y[:3000].contiguous())
    K.applyDiffKT(X, X, X)
    assert nat.WORKSPACE.get(1).numel() <= 64 << 20
    Z = X[:5000].contiguous()
    a = K.applyK(Z, Z)
    b = K.applyK(Z, Z, firstVar=Z.clone())
    assert float((a - b).norm() / b.norm()) < 1e-13

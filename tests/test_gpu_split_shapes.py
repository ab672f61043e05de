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


@pytest.mark.parametrize('dtype,tol', [('float32', 2e-5), ('float64', 1e-12)])
@pytest.mark.parametrize('n,m', [(1, 1), (1, 700), (31, 33), (63, 128), (64, 129), (129, 1), (256, 127), (257, 511),
                                 (1025, 2000), (3000, 1500), (5000, 5000)])
def test_ordered_sums_split_and_whole(n, m, dtype, tol):
    """The ordered-pair operators at the edges of the split shapes' blocks (32 RT targets), on both sides of the rule
    that chooses them, against the oracle; tolerances of the operator tests."""
    import oracle as O
    from base.kernelFunctions import Kernel
    rng = np.random.default_rng(1000 * n + m)
    y, x = rng.normal(size=(n, 3)), rng.normal(size=(m, 3))
    a, p = rng.normal(size=(m, 3)), rng.normal(size=(n, 3))
    K = Kernel(name='gauss', sigma=0.7)
    K.pk_dtype = dtype

    def close(got, ref):
        return np.linalg.norm(got - ref) <= tol * np.linalg.norm(ref) + 0.05 * tol * np.sqrt(ref.size)

    assert close(K.applyK(x, a, firstVar=y), O.apply_k(y, x, a, 0.7))
    assert close(K.applyDiffKT(x, p, a, firstVar=y), O.apply_diff_kt(y, x, p, a, 0.7))
    assert close(K.applyDivergence(x, a, firstVar=y).ravel(), np.ravel(O.apply_divergence(y, x, a, 0.7)))
    ay, ax = rng.normal(size=n), rng.normal(size=m)
    kt = O.apply_k_tensor(y, x, ay, ax, p, a, 0.7)
    assert close(K.applyKTensor(x, ay, ax, p, a, firstVar=y).ravel(), np.ravel(kt))
    q = rng.normal(size=(n, 3))
    assert close(K.applyDDiffK11and12(y, p, q, p), O.apply_ddiff_k11and12(y, p, q, p, 0.7))
    assert close(K.applyDiffK1and2(y, p, q), O.apply_diff_k1and2(y, p, q, 0.7))


@pytest.mark.parametrize('nf,nf1', [(1, 1), (127, 1), (128, 129), (129, 640), (257, 255), (1025, 3000), (3000, 700),
                                    (5120, 5119)])
def test_energies_once_per_unordered_self_pair(nf, nf1):
    """Varifold, current and measure energies and norms of meshes whose face counts end inside a tile, a row block and
    the self part of the sources, against the oracle. Tolerances of the surface tests: 1e-6 of the energy's two norms
    in FP32, 1e-11 in FP64."""
    import oracle as O
    from base.kernelFunctions import Kernel
    from base.surfaceDistances import SurfaceDataTerm
    from base.syntheticShapes import bumpy_ellipsoid, icosphere
    v, f = icosphere(4)
    x, x1 = bumpy_ellipsoid(v, seed=3), bumpy_ellipsoid(v, seed=4)
    f0, f1 = f[:nf], f[::-1][:nf1].copy()
    for kind in ('varifold', 'current', 'measure'):
        norm0 = {'varifold': O.varifold_norm0, 'current': O.current_norm0, 'measure': O.measure_norm0}[kind]
        ndef = {'varifold': O.varifold_norm_def, 'current': O.current_norm_def, 'measure': O.measure_norm_def}[kind]
        ref, ref0 = ndef(x, f0, x1, f1, 0.3), norm0(x1, f1, 0.3)
        size = abs(ref0) + norm0(x, f0, 0.3)
        for dtype, tol in (('float32', 1e-6), ('float64', 1e-11)):
            Kd = Kernel(name='gauss', sigma=0.3)
            Kd.pk_dtype = dtype
            e = SurfaceDataTerm(f0, x1, f1, Kd, kind=kind, nv=x.shape[0]).energy(x, with_norm0=True).tolist()
            assert abs(e[0] - ref) <= tol * size and abs(e[1] - ref0) <= tol * size, (kind, dtype)


@pytest.mark.parametrize('name', ['gauss', 'laplacian'])
@pytest.mark.parametrize('n', [1, 700, 3000, 9000, 17000])
def test_sums_far_from_the_coordinate_origin(n, name):
    """Self-sums and a shooting step without a caller's origin on points 1,000 widths from 0, one of them much further:
    the same FP32 accuracy as at 0 (2e-5 relative, Laplacian 3e-5), against the FP64 sums of the shifted points."""
    import torch
    from base import pointEvolution as evol
    from base.kernelFunctions import Kernel
    rng = np.random.default_rng(n)
    X = torch.from_numpy(rng.normal(size=(n, 3))).cuda()
    A = torch.from_numpy(rng.normal(size=(n, 3))).cuda()
    if 1 < n <= 16384:             # larger sets centre a block on its box, which one far point stretches
        X[0, 1] = 2.0e5            # the first point of the first block
    off = torch.tensor([800.0, -500.0, 300.0], dtype=torch.float64, device='cuda')
    K, K64 = Kernel(name=name, sigma=0.8, order=3), Kernel(name=name, sigma=0.8, order=3)
    K.pk_dtype, K64.pk_dtype = 'float32', 'float64'
    tol = 2e-5 if name == 'gauss' else 3e-5
    ka, za = K64.applyK(X, A), -K64.applyDiffKT(X, A, A)

    def close(a, b):
        return float((a - b).norm()) <= tol * float(b.norm()) + 1e-6 * n ** 0.5

    assert close(K.applyK(X + off, A), ka)
    xt, at = evol.shoot_second_order(X + off, A, K, 1.0)
    assert close(xt[1] - xt[0], ka)
    assert close(at[1] - A, za)

"""The origin that a block of a small set takes for itself when the caller gives none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _errors(X, A, P, B, name, origin):
    import torch
    from base import _native as nat
    from base import pointEvolution as evol
    from base.kernelFunctions import Kernel
    out = {}
    for dtype, o in (('float32', origin), ('float64', nat.centroid(X))):
        K = Kernel(name=name, sigma=1.0, order=3) if name == 'laplacian' else Kernel(name=name, sigma=1.0)
        K.pk_dtype = dtype
        xt, at = evol.shoot_second_order(X, A, K, 1.0, origin=o)
        px, pa, _ = evol.second_order_adjoint(torch.stack([X, X]), torch.stack([A, A]), P, B, K, 1.0, origin=o,
                                              with_da0=False)
        f1, f0 = evol.first_order_gradient(torch.stack([X, X]), A[None].contiguous(), P, K, 0.5, euclidean=True,
                                           origin=o)
        out[dtype] = [K._apply_k(X, X, A, 1.0, o), xt[1] - X, at[1] - A, px[0] - P, pa[0] - B, f1[0] - P, f0[0]]
    return [float((a - b).norm() / b.norm()) for a, b in zip(out['float32'], out['float64'])]


@pytest.mark.parametrize('name', ['gauss', 'laplacian'])
@pytest.mark.parametrize('n', [700, 1300, 2600, 5000, 8000])
def test_scattered_sets_are_as_accurate_as_about_their_centroid(n, name):
    """Points of a cube of 32 widths in random order: the FP32 errors of self-sums and steps without an origin against
    those about the centroid. The rounding of a coordinate grows with its distance from the origin; the middle of a block
    lies within an eighth of the half extent from the centre in the mean square, which adds 3 / 8^2 / 2 = 2.3% to the
    error. Bound: 10% on the geometric mean of seven sums over three sets (their errors are sums of thousands of
    roundings), where an origin at half the extent adds 30%."""
    import torch
    ratios = []
    for seed in range(3):
        r = np.random.default_rng(100 * seed + n)
        X = torch.from_numpy(r.uniform(-16, 16, size=(n, 3))).cuda()
        A, P, B = (torch.from_numpy(r.normal(size=(n, 3))).cuda() for _ in range(3))
        own = _errors(X, A, P, B, name, None)
        given = _errors(X, A, P, B, name, X.mean(0).tolist())
        ratios += [a / b for a, b in zip(own, given)]
    assert float(np.exp(np.mean(np.log(ratios)))) < 1.1, np.round(ratios, 2)


@pytest.mark.parametrize('far', [1e3, -2e5, 1e30])
@pytest.mark.parametrize('where', [0, 1, 20, 63, 64, 100, 127])
def test_one_far_point_does_not_move_a_block(far, where):
    """At any place of a block: the other points' sums are those of the set without it, whose blocks are as close to
    their points. Bound 2e-5, that of the FP32 kernel sums; the far point is beyond the kernel's reach."""
    import torch
    from base.kernelFunctions import Kernel
    r = np.random.default_rng(where)
    x, a = r.normal(size=(700, 3)) + 40.0, r.normal(size=(700, 3))
    x[where, 1] = far
    K, K64 = Kernel(name='gauss', sigma=0.5), Kernel(name='gauss', sigma=0.5)
    K.pk_dtype, K64.pk_dtype = 'float32', 'float64'
    X, A = torch.from_numpy(x).cuda(), torch.from_numpy(a).cuda()
    got, ref = K.applyK(X, A), K64.applyK(X, A)
    keep = torch.arange(700, device='cuda') != where
    assert float((got - ref)[keep].norm()) < 2e-5 * float(ref[keep].norm())
    assert bool(torch.isfinite(got).all())


@pytest.mark.parametrize('n', [1, 2, 3, 4, 5, 33, 65, 66, 67, 68])
def test_blocks_of_few_points(n):
    """Fewer points than groups in the last (or only) block, far from the coordinate origin."""
    import torch
    from base.kernelFunctions import Kernel
    r = np.random.default_rng(n)
    X = torch.from_numpy(r.normal(size=(n, 3)) - 5.0e4).cuda()
    A = torch.from_numpy(r.normal(size=(n, 3))).cuda()
    K, K64 = Kernel(name='gauss', sigma=0.5), Kernel(name='gauss', sigma=0.5)
    K.pk_dtype, K64.pk_dtype = 'float32', 'float64'
    got, ref = K.applyK(X, A), K64.applyK(X, A)
    assert float((got - ref).norm()) < 2e-5 * float(ref.norm())


@pytest.mark.parametrize('dtype', ['float32', 'float64'])
def test_far_points_at_the_ends_and_the_middle_of_a_block(dtype):
    """The three points that a block's reference is taken from may all be far ones (2e5 widths): the others' sums stay
    those of the kernel tests (FP32 2e-5; FP64 coordinates at 2e5 widths round at 2^-53 x 2e5 of a width, 1e-10)."""
    import torch
    import oracle as O
    from base.kernelFunctions import Kernel
    r = np.random.default_rng(5)
    x, a = r.normal(size=(640, 3)), r.normal(size=(640, 3))
    far = np.zeros(640, dtype=bool)
    for b in (32, 64, 128):
        for k in range(0, 640, b):
            far[[k, k + (b - 1) // 2, k + b - 1]] = k % 256 == 0
    x[far, 0] += 2.0e5
    K = Kernel(name='gauss', sigma=1.0)
    K.pk_dtype = dtype
    got, ref = K.applyK(x, a), O.apply_k(x, x, a, 1.0)
    tol = 2e-5 if dtype == 'float32' else 1e-10
    assert np.linalg.norm((got - ref)[~far]) < tol * np.linalg.norm(ref[~far])


@pytest.mark.parametrize('run', [2, 5, 6, 8])
@pytest.mark.parametrize('start', [0, 3, 12, 24])
@pytest.mark.parametrize('n', [300, 2000])
def test_a_run_of_far_points_does_not_move_a_block(n, start, run):
    """Far points in a row (1e9 and more, apart from each other), up to a quarter of the points that a block's origin is
    taken from (32, or all of a shorter block): the FP64 sums of the others are those of
    points within 16 of their origin. Coordinates of 27 widths' scale round at 27 x 2^-53, differences at 1.2e-14 at most,
    and a term 2^-|d|^2 with |d| up to 5 at 2 x 5 x ln 2 of that: below 1e-13; bound 2e-13. About an origin that a far point
    has moved by a sixteenth they would round at 1e-8."""
    import torch
    from base.kernelFunctions import Kernel
    r = np.random.default_rng(start + 100 * run)
    x, a = r.uniform(0, 16, size=(n, 3)), r.normal(size=(n, 3))
    far = np.zeros(n, dtype=bool)
    for b in range(0, n, 64):
        far[b + start:b + start + min(run, min(n - b, 32) // 4)] = True
    x[far, 0] += 1.0e9 * (1 + np.arange(int(far.sum())))
    X, A = torch.from_numpy(x).cuda(), torch.from_numpy(a).cuda()
    got = Kernel(name='gauss', sigma=0.5).applyK(X, A)[torch.from_numpy(~far).cuda()]
    near, an = X[torch.from_numpy(~far).cuda()], A[torch.from_numpy(~far).cuda()]
    ref = torch.exp(-2.0 * ((near[:, None] - near[None]) ** 2).sum(-1)) @ an
    assert float((got - ref).norm()) < 2e-13 * float(ref.norm())

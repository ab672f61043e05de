"""Timing cases of the point-set path: what a registration user calls, at the sizes users have.

`listed()` names the cases that are timed, `draw(rng)` gives further ones of the same ranges, `prepare` makes a
case's inputs on the GPU (host arrays where the entry point takes host arrays), `run` makes one pass through the
public entry points, `work` counts what a pass cannot do without and `exact` evaluates the same formulas in float64
with plain torch, without this package's kernels.

Kernel sums asked for in 'float32' carry float32 precision, whatever the type of the array they are returned in; a
program that asks for them keeps the results in float32, and so does `run`. Sums in 'float64' stay float64.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), 'py-lddmm_b200'))

from base import pointEvolution as evol                                                     # noqa: E402
from base.autograd import geodesic_registration_loss                                        # noqa: E402
from base.kernelFunctions import Kernel                                                     # noqa: E402
from base.learnedProposal import HIDDEN, IN_DIM, MomentumProposal, N_FEATURES, N_OUT, OUT_DIM  # noqa: E402
from base.surfaceDistances import SurfaceDataTerm, varifoldNormDef, varifoldNormGradient    # noqa: E402
from base.surfaceMatching import SecondOrderSurfaceMatching                                 # noqa: E402
from base.surfaces import Surface                                                           # noqa: E402
from base.syntheticShapes import bumpy_ellipsoid, icosphere                                 # noqa: E402


def listed():
    return [
        # the drop-in call of a script on a small landmark set: numpy in, numpy out, the default precision
        {'name': 'applyk_host_642_f64', 'do': 'applyk', 'n': 642, 'sigma': 0.5, 'dtype': 'float64', 'host': True},
        # velocity of a full-resolution surface (icosphere level 6), the benchmark's kernel sum
        {'name': 'applyk_40962_f32', 'do': 'applyk', 'n': 40962, 'sigma': 0.25, 'dtype': 'float32', 'host': False},
        # velocity of a surface's momenta at scattered points (a point set or grid nodes carried along), ragged sizes
        {'name': 'points_30011_f32', 'do': 'points', 'n': 30011, 'm': 20481, 'sigma': 0.25, 'dtype': 'float32'},
        # gradient of geodesic shooting at the coarse level of a registration (level 4, 10 steps)
        {'name': 'geodesic_2562_f32', 'do': 'geodesic', 'n': 2562, 'sigma': 0.5, 'dtype': 'float32', 'steps': 10},
        # the same at full resolution (level 6)
        {'name': 'geodesic_40962_f32', 'do': 'geodesic', 'n': 40962, 'sigma': 0.5, 'dtype': 'float32', 'steps': 10},
        # the same in float64, the kernels' default precision (level 5)
        {'name': 'geodesic_10242_f64', 'do': 'geodesic', 'n': 10242, 'sigma': 0.5, 'dtype': 'float64', 'steps': 10},
        # first-order landmark matching with the Laplacian kernel: trajectory, covector and gradient
        {'name': 'landmark_lap_10242_f32', 'do': 'landmark', 'n': 10242, 'sigma': 0.5, 'dtype': 'float32',
         'steps': 10, 'order': 3},
        # data term of a full-resolution registration: varifold energy and gradient, level-6 faces on both sides
        {'name': 'varifold_81920_f32', 'do': 'varifold', 'nu': 0, 'nv': 6, 'nu1': 0, 'nv1': 6, 'sigma': 0.2,
         'dtype': 'float32', 'host': False},
        # the same through the reference's functions on two scanned-like meshes of different, odd face counts
        {'name': 'varifold_host_2990_f64', 'do': 'varifold', 'nu': 65, 'nv': 23, 'nu1': 57, 'nv1': 31, 'sigma': 0.3,
         'dtype': 'float64', 'host': True},
        # a differentiable registration objective with its backward pass (level 5, checkpointed every 5 steps)
        {'name': 'loss_10242_f32', 'do': 'loss', 'nu': 0, 'nv': 5, 'nu1': 0, 'nv1': 5, 'sigma': 0.5,
         'sigma_dist': 0.2, 'dtype': 'float32', 'steps': 10},
        # the start of a registration, whole: matching object, three BFGS iterations, deformed surface (level 4)
        {'name': 'registration_2562_f32', 'do': 'registration', 'nu': 0, 'nv': 4, 'nu1': 0, 'nv1': 4, 'sigma': 0.5,
         'sigma_dist': 0.3, 'dtype': 'float32', 'steps': 10, 'iters': 3},
        # one training step of the momentum network on a batch of 16 level-4 pairs
        {'name': 'proposal_41984', 'do': 'proposal', 'n': 41984},
    ]


def draw(rng):
    """One more case: a kind of call, then its sizes (log-uniform over the kind's range), width and options."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def rings(lo, hi):                                  # a sphere of nu x nv rings with about lo..hi faces
        f = size(lo, hi)
        nv = max(3, int(math.sqrt(f / 4) * rng.uniform(0.6, 1.2)))
        return max(5, f // (2 * nv)), nv

    sig = round(rng.uniform(0.2, 0.6), 3)
    do = rng.choice(('applyk', 'applyk', 'points', 'geodesic', 'geodesic', 'geodesic', 'landmark', 'varifold',
                     'varifold', 'loss', 'registration', 'proposal'))
    f64 = rng.random() < 0.35
    dt = 'float64' if f64 else 'float32'
    if do == 'applyk':
        return {'do': do, 'n': size(100, 40000), 'sigma': sig, 'dtype': dt, 'host': rng.random() < 0.5}
    if do == 'points':
        return {'do': do, 'n': size(200, 40000), 'm': size(200, 40000), 'sigma': sig, 'dtype': dt}
    if do == 'geodesic':
        return {'do': do, 'n': size(200, 10000 if f64 else 40000), 'sigma': sig, 'dtype': dt,
                'steps': rng.choice((5, 10))}
    if do == 'landmark':
        c = {'do': do, 'n': size(200, 10000 if f64 else 30000), 'sigma': sig, 'dtype': dt,
             'steps': rng.choice((5, 10))}
        return dict(c, order=rng.choice((1, 2, 3, 4))) if rng.random() < 0.7 else c
    if do == 'varifold':
        nu, nv = rings(300, 20000 if f64 else 80000)
        nu1, nv1 = rings(300, 20000 if f64 else 80000)
        return {'do': do, 'nu': nu, 'nv': nv, 'nu1': nu1, 'nv1': nv1, 'sigma': round(rng.uniform(0.1, 0.4), 3),
                'dtype': dt, 'host': rng.random() < 0.4}
    if do in ('loss', 'registration'):
        nu, nv = rings(300, 20000)
        nu1, nv1 = rings(300, 20000)
        c = {'do': do, 'nu': nu, 'nv': nv, 'nu1': nu1, 'nv1': nv1, 'sigma': round(rng.uniform(0.4, 0.6), 3),
             'sigma_dist': round(rng.uniform(0.2, 0.4), 3), 'dtype': 'float32', 'steps': rng.choice((5, 10))}
        return dict(c, iters=3) if do == 'registration' else c
    return {'do': 'proposal', 'n': 64 * size(4, 640)}


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=16)
def _sphere(nu, nv):
    """Unit sphere mesh (vertices, faces): the icosphere of level nv (nu = 0), or nv rings of nu vertices and two
    poles (2 nu nv faces), rows in order as a scanner or an iso-surface extraction leaves them."""
    if nu == 0:
        return icosphere(nv)
    th = np.pi * np.arange(1, nv + 1) / (nv + 1)
    ph = 2 * np.pi * np.arange(nu) / nu
    ring = np.stack([np.sin(th)[:, None] * np.cos(ph), np.sin(th)[:, None] * np.sin(ph),
                     np.repeat(np.cos(th)[:, None], nu, 1)], 2).reshape(-1, 3)
    v = np.concatenate([[[0., 0., 1.]], ring, [[0., 0., -1.]]])
    i, j = np.arange(nu), (np.arange(nu) + 1) % nu
    faces = [np.stack([0 * i, 1 + i, 1 + j], 1)]
    for r in range(nv - 1):
        a, b = 1 + r * nu, 1 + (r + 1) * nu
        faces.append(np.stack([np.stack([a + i, b + i, b + j], 1), np.stack([a + i, b + j, a + j], 1)], 1)
                     .reshape(-1, 3))
    a = 1 + (nv - 1) * nu
    faces.append(np.stack([a + i, 0 * i + nu * nv + 1, a + j], 1))
    return v, np.concatenate(faces).astype(np.int64)


@functools.lru_cache(maxsize=16)
def _unit_points(n):
    """n points of the unit sphere: the icosphere with n vertices if there is one, else a spiral."""
    for level in range(8):
        if n == 10 * 4 ** level + 2:
            return icosphere(level)[0]
    z = 1 - (2 * np.arange(n) + 1) / n
    ph = np.pi * (1 + 5 ** 0.5) * np.arange(n)
    s = np.sqrt(1 - z * z)
    return np.stack([s * np.cos(ph), s * np.sin(ph), z], 1)


def _source(sphere, seed):
    """A surface near the unit sphere; another seed is another surface."""
    return bumpy_ellipsoid(sphere, n_bumps=6, amplitude=0.03, width=0.35, seed=2 * seed + 1, axes=(1.0, 1.05, 0.95))


def _target(sphere, seed):
    return bumpy_ellipsoid(sphere, seed=2 * seed)


def _field(x, gen, terms=8, freq=2.5):
    """A smooth random vector field at x (N,3)."""
    w = torch.randn((3, terms), generator=gen, device='cuda', dtype=torch.float64) * freq
    ph = torch.rand((1, terms), generator=gen, device='cuda', dtype=torch.float64) * 2 * math.pi
    c = torch.randn((terms, 3), generator=gen, device='cuda', dtype=torch.float64)
    return torch.sin(x @ w + ph) @ c


def _momenta(case, x, gen, speed=0.3):
    """Smooth momenta with an initial speed of about `speed` (estimated from every k-th point as source)."""
    a = _field(x, gen)
    k = max(1, x.shape[0] // 512)
    v = _radial(case, torch.cdist(x, x[::k]))[0] @ a[::k] * k
    return (a * (speed / v.norm(dim=1).max())).contiguous()


def _kernel(case):
    if case.get('order') is not None:
        K = Kernel(name='laplacian', sigma=case['sigma'], order=case['order'])
    else:
        K = Kernel(name='gauss', sigma=case['sigma'])
    K.pk_dtype = case['dtype']
    return K


def _gen(seed):
    return torch.Generator(device='cuda').manual_seed(1000003 * int(seed) + 17)


def _dist_kernel(case, key='sigma'):
    Kd = Kernel(name='gauss', sigma=case[key])
    Kd.pk_dtype = case['dtype']
    return Kd


def prepare(case, seed):
    do, gen = case['do'], _gen(seed)
    st = {'case': case}
    if do in ('applyk', 'points', 'geodesic', 'landmark'):
        n = case['m'] if do == 'points' else case['n']
        x = torch.from_numpy(_source(_unit_points(n), seed)).cuda()
        a = _momenta(case, x, gen)
        st.update(K=_kernel(case), x=x, a=a)
        if do == 'applyk' and case['host']:
            st.update(x=x.cpu().numpy(), a=a.cpu().numpy())
        elif do == 'points':
            u = torch.rand((case['n'], 3), generator=gen, device='cuda', dtype=torch.float64)
            st['y'] = 2.6 * u - 1.3
        elif do == 'geodesic':
            st['px1'] = 0.05 * _field(x, gen) / math.sqrt(x.shape[0])
            st['pa1'] = torch.zeros_like(x)
        elif do == 'landmark':
            T = case['steps']
            st['at'] = torch.stack([a * (1 - 0.5 * t / T) for t in range(T)]).contiguous()
            st['px1'] = 0.05 * _field(x, gen) / math.sqrt(x.shape[0])
        return st
    if do == 'proposal':
        n = case['n']
        F = torch.zeros((n, IN_DIM), device='cuda')
        F[:, :N_FEATURES] = 0.5 * torch.randn((n, N_FEATURES), generator=gen, device='cuda')
        W = torch.randn((N_FEATURES, N_OUT), generator=gen, device='cuda') / math.sqrt(N_FEATURES)
        st.update(F=F.to(torch.bfloat16), target=torch.tanh(F[:, :N_FEATURES] @ W).contiguous(),
                  model=MomentumProposal(seed=seed))
        return st
    sph, faces = _sphere(case['nu'], case['nv'])
    sph1, faces1 = _sphere(case['nu1'], case['nv1'])
    x, x1 = _source(sph, seed), _target(sph1, seed)
    if do == 'varifold':
        Kd = _dist_kernel(case)
        if case['host']:
            st.update(surf=Surface(surf=(faces, x)), surf1=Surface(surf=(faces1, x1)), Kd=Kd)
        else:
            st.update(term=SurfaceDataTerm(faces, x1, faces1, Kd, kind='varifold', nv=x.shape[0]),
                      x=torch.from_numpy(x).cuda())
    elif do == 'loss':
        X = torch.from_numpy(x).cuda()
        st.update(K=_kernel(case), x=X, a=_momenta(case, X, gen, 0.2),
                  term=SurfaceDataTerm(faces, x1, faces1, _dist_kernel(case, 'sigma_dist'), kind='varifold',
                                       nv=x.shape[0]))
    else:
        st.update(surf=Surface(surf=(faces, x)), surf1=Surface(surf=(faces1, x1)))
    return st


# ---------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------
def _keep(case, v):
    """Results as the program keeps them: float32 for sums in float32."""
    if v is None or case['dtype'] == 'float64':
        return v
    return v.float() if isinstance(v, torch.Tensor) else np.asarray(v, dtype=np.float32)


def run(st):
    case = st['case']
    do = case['do']
    if do == 'applyk':
        return _keep(case, st['K'].applyK(st['x'], st['a']))
    if do == 'points':
        return _keep(case, st['K'].applyK(st['x'], st['a'], firstVar=st['y']))
    if do == 'geodesic':
        r = evol.secondOrderGradient(st['x'], st['a'], st['px1'], st['pa1'], st['K'], 1.0 / case['steps'])
        return {k: _keep(case, r[k]) for k in ('da0', 'xt', 'at', 'pxt', 'pat')}
    if do == 'landmark':
        dat, xt, pxt = evol.landmarkHamiltonianGradient(st['x'], st['at'], st['px1'], st['K'], 1.0, getCovector=True)
        return {'dat': _keep(case, dat), 'xt': _keep(case, xt), 'pxt': _keep(case, pxt)}
    if do == 'varifold':
        if case['host']:
            e = varifoldNormDef(st['surf'], st['surf1'], st['Kd'])
            g = varifoldNormGradient(st['surf'], st['surf1'], st['Kd'])
        else:
            e = st['term'].energy(st['x'])[:1]
            g = st['term'].gradient(st['x'])
        return {'energy': _keep(case, e), 'gradient': _keep(case, g)}
    if do == 'loss':
        x, a = st['x'].detach().requires_grad_(), st['a'].detach().requires_grad_()
        loss = geodesic_registration_loss(x, a, st['K'], st['term'], 1.0 / case['steps'])
        loss.backward()
        return {'loss': _keep(case, loss.detach()), 'dx0': _keep(case, x.grad), 'da0': _keep(case, a.grad)}
    if do == 'registration':
        opts = dict(maxIter=case['iters'], KparDiff=('gauss', case['sigma']), KparDist=('gauss', case['sigma_dist']),
                    sigmaError=1.0, errorType='varifold', pk_dtype=case['dtype'], algorithm='bfgs',
                    timeStep=1.0 / case['steps'], verb=False, affine='none')
        f = SecondOrderSurfaceMatching(Template=st['surf'], Target=st['surf1'], options=opts)
        f.optimizeMatching()
        return {'a0': _keep(case, f.control['a0']), 'deformed': _keep(case, f.fvDef.vertices)}
    model = st['model']
    loss, grads = model.gradients(st['F'], st['target'], case['n'])
    model.adam(grads)
    return {'loss': loss, 'grads': grads, 'weights': list(model.W), 'bias': list(model.b)}


# ---------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------
def _faces(nu, nv):
    return 20 * 4 ** nv if nu == 0 else 2 * nu * nv


def _verts(nu, nv):
    return 10 * 4 ** nv + 2 if nu == 0 else nu * nv + 2


def work(case):
    """Bytes: float64 inputs once, float64 outputs once. Flops: additions and multiplications of each pair sum, an
    unordered pair of a self-sum evaluated once and credited to both points, an exponential counted as one."""
    do = case['do']
    D = 24                                                                            # bytes of a point
    if do == 'applyk':
        n = case['n']
        return {'bytes': 3 * D * n, 'flops': n * n / 2 * (9 + 12)}
    if do == 'points':
        return {'bytes': D * (2 * case['n'] + 2 * case['m']), 'flops': case['n'] * case['m'] * (9 + 6.0)}
    if do == 'geodesic':
        n, T = case['n'], case['steps']
        return {'bytes': D * n * (4 + 4 * (T + 1) + 1), 'flops': n * n / 2 * (T * (9 + 6 + 24) + T * (9 + 70) + 21)}
    if do == 'landmark':
        n, T = case['n'], case['steps']
        e = 9 + (3 * case['order'] if case.get('order') else 0)
        return {'bytes': D * n * (2 + T + 2 * (T + 1) + T), 'flops': n * n / 2 * (T * (e + 12) + T * (e + 12 + 12))}
    if do == 'proposal':
        n, p = case['n'], IN_DIM * HIDDEN + 2 * HIDDEN * HIDDEN + HIDDEN * OUT_DIM
        return {'bytes': n * (2 * IN_DIM + 4 * N_OUT) + 24 * p, 'flops': 2.0 * n * (3 * p - IN_DIM * HIDDEN)}
    f, f1 = _faces(case['nu'], case['nv']), _faces(case['nu1'], case['nv1'])
    v, v1 = _verts(case['nu'], case['nv']), _verts(case['nu1'], case['nv1'])
    pairs = f * f / 2 + f * f1
    energy, grad = pairs * (9 + 6 + 4), (f * f / 2 * 2 + f * f1) * 18 + pairs * (9 + 6 + 4)
    mesh = D * (v + f + v1 + f1)
    if do == 'varifold':
        return {'bytes': 2 * mesh + D * v + 8, 'flops': energy + grad}
    T = case['steps']
    step = v * v / 2
    one = step * (T * 39 + T * 79 + 21) + energy + grad
    traj = D * v * (4 + 4 * (T + 1))
    if do == 'loss':
        return {'bytes': mesh + traj, 'flops': one + step * 33}
    return {'bytes': mesh + case['iters'] * traj, 'flops': case['iters'] * one}


# ---------------------------------------------------------------------------------------------------------------
# the same results in float64 with plain torch
# ---------------------------------------------------------------------------------------------------------------
# P0 of the Laplacian kernel P0(u) exp(-u), u = r / sigma, by order; P1 = (P0 - P0') / u, the factor of -(y-x)/sigma^2
# in its gradient (zero for order 0)
_LAP = {1: ([1, 1], [1]), 2: ([1, 1, 1 / 3], [1 / 3, 1 / 3]), 3: ([1, 1, 0.4, 1 / 15], [0.2, 0.2, 1 / 15]),
        4: ([1, 1, 3 / 7, 2 / 21, 1 / 105], [1 / 7, 1 / 7, 2 / 35, 1 / 105])}


def _radial(case, r):
    """(K, K1) at distances r: kernel values and the factor of -(y - x)/sigma^2 in the gradient."""
    if case.get('order') is None:
        e = torch.exp(-0.5 * (r / case['sigma']) ** 2)
        return e, e
    u = r / case['sigma']
    e = torch.exp(-u)
    p0, p1 = (sum(c * u ** k for k, c in enumerate(cs)) for cs in _LAP[case['order']])
    return p0 * e, p1 * e


def _rows(n, m=None):
    m = n if m is None else m
    step = max(1, int(4e8 // (8 * max(1, m))))
    return [slice(i, min(n, i + step)) for i in range(0, n, step)]


def _dist(y, x):
    d2 = (y * y).sum(1, keepdim=True) + (x * x).sum(1) - 2 * (y @ x.T)
    near = d2 < 1e-4                                   # the differences themselves where the expansion cancels
    i, j = near.nonzero(as_tuple=True)
    d2[i, j] = ((y[i] - x[j]) ** 2).sum(1)
    return d2.clamp_min(0).sqrt()


def _k(case, y, x, a):
    return torch.cat([_radial(case, _dist(y[s], x))[0] @ a for s in _rows(y.shape[0], x.shape[0])])


def _pull(w, y, x):
    """sum_l w_kl (y_k - x_l)."""
    return y * w.sum(1, keepdim=True) - w @ x


def _so_forward(case, x, a, dt):
    v, z = torch.empty_like(x), torch.empty_like(x)
    for s in _rows(x.shape[0]):
        e, e1 = _radial(case, _dist(x[s], x))
        v[s] = e @ a
        z[s] = _pull(e1 * (a[s] @ a.T), x[s], x) / case['sigma'] ** 2
    return x + dt * v, a + dt * z


def _so_adjoint(case, x, a, px, pa, dt):
    is2 = 1 / case['sigma'] ** 2
    zx, za = torch.empty_like(x), torch.empty_like(x)
    for s in _rows(x.shape[0]):
        e = _radial(case, _dist(x[s], x))[0]
        dq = ((x[s] * pa[s]).sum(1, keepdim=True) + (x * pa).sum(1) - x[s] @ pa.T - pa[s] @ x.T) * e
        na = a[s] @ a.T
        zx[s] = -is2 * _pull(e * (px[s] @ a.T + a[s] @ px.T), x[s], x) \
            - (is2 * is2 * _pull(na * dq, x[s], x) - is2 * _pull(na * e, pa[s], pa))
        za[s] = e @ px + is2 * (dq @ a)
    return px + dt * zx, pa + dt * za


def _varifold(xdef, faces, x1, faces1, sigma, grad=True):
    """(|def|^2 - 2 <def, tgt>, its gradient at the vertices, |tgt|^2)."""
    def geometry(v, f):
        p, q, r = v[f[:, 0]], v[f[:, 1]], v[f[:, 2]]
        s = torch.linalg.cross(q - p, r - p) / 2
        return (p + q + r) / 3, s, ((s * s).sum(1, keepdim=True) + 1e-10).sqrt()

    xdef = xdef.detach().requires_grad_(grad)
    c, s, ar = geometry(xdef, faces)
    c1, s1, ar1 = geometry(x1, faces1)
    C, S, A = c.detach(), s.detach(), ar.detach()
    dC, dS, tot = torch.zeros_like(C), torch.zeros_like(S), 0.0
    case = {'sigma': sigma}

    def norm2(cs, ss, aa, co, so, ao, weight, dc, ds):
        t = 0.0
        n, no = ss / aa, so / ao
        for r in _rows(cs.shape[0], co.shape[0]):
            g = n[r] @ no.T
            e = _radial(case, _dist(cs[r], co))[0] * ao.T
            g2 = e * g * g
            w = e + g2
            t = t + (aa[r, 0] * w.sum(1)).sum()
            if dc is not None:
                dc[r] += -2 * weight * aa[r] * _pull(w, cs[r], co) / sigma ** 2
                ds[r] += 2 * weight * ((e - g2).sum(1, keepdim=True) * n[r] + 2 * (e * g) @ no)
        return t

    tot = norm2(C, S, A, C, S, A, 1.0, dC if grad else None, dS) \
        - 2 * norm2(C, S, A, c1, s1, ar1, -1.0 if grad else 0.0, dC if grad else None, dS)
    px = torch.autograd.grad((c * dC).sum() + (s * dS).sum(), xdef)[0] if grad else None
    return tot, px, norm2(c1, s1, ar1, c1, s1, ar1, 0.0, None, None)


def exact(case, seed):
    if case['do'] == 'registration':      # its line search takes decisions: no value of its own in 64 bits
        return None
    st = prepare(case, seed)
    do = case['do']
    if do in ('applyk', 'points'):
        x, a = (torch.as_tensor(st[k]).cuda() for k in ('x', 'a'))
        r = _k(case, st.get('y', x), x, a)
        return r.cpu().numpy() if case.get('host') else r
    if do == 'geodesic':
        T, dt = case['steps'], 1.0 / case['steps']
        xt, at = [st['x']], [st['a']]
        for _ in range(T):
            x, a = _so_forward(case, xt[-1], at[-1], dt)
            xt.append(x)
            at.append(a)
        pxt, pat = [st['px1']], [st['pa1']]
        for t in range(T - 1, -1, -1):
            px, pa = _so_adjoint(case, xt[t], at[t], pxt[0], pat[0], dt)
            pxt.insert(0, px)
            pat.insert(0, pa)
        return {'da0': _k(case, xt[0], xt[0], at[0]) - pat[0], 'xt': torch.stack(xt), 'at': torch.stack(at),
                'pxt': torch.stack(pxt), 'pat': torch.stack(pat)}
    if do == 'landmark':
        T, dt, w, at = case['steps'], 1.0 / case['steps'], 1.0, st['at']
        xt = [st['x']]
        for t in range(T):
            xt.append(xt[-1] + dt * _k(case, xt[-1], xt[-1], at[t]))
        pxt = [st['px1']]
        for t in range(T - 1, -1, -1):
            x, a, p = xt[t], at[t], pxt[0]
            z = torch.empty_like(x)
            for s in _rows(x.shape[0]):
                c = p[s] @ a.T + a[s] @ (p - 2 * w * a).T
                z[s] = -_pull(_radial(case, _dist(x[s], x))[1] * c, x[s], x) / case['sigma'] ** 2
            pxt.insert(0, p + dt * z)
        pxt = torch.stack(pxt)
        return {'dat': 2 * w * at - pxt[1:], 'xt': torch.stack(xt), 'pxt': pxt}
    if do == 'varifold':
        if case['host']:
            x, f, x1, f1 = (torch.as_tensor(v).cuda() for v in (st['surf'].vertices, st['surf'].faces,
                                                                st['surf1'].vertices, st['surf1'].faces))
        else:
            x, f, x1, f1 = st['x'], st['term'].faces, st['term'].x1, st['term'].faces1
        e, g, _ = _varifold(x, f, x1, f1, case['sigma'])
        if case['host']:
            return {'energy': float(e), 'gradient': g.cpu().numpy()}
        return {'energy': e.reshape(1), 'gradient': g}
    if do == 'loss':
        T, dt = case['steps'], 1.0 / case['steps']
        xt, at = [st['x']], [st['a']]
        for _ in range(T):
            x, a = _so_forward(case, xt[-1], at[-1], dt)
            xt.append(x)
            at.append(a)
        e, px, e1 = _varifold(xt[-1], st['term'].faces, st['term'].x1, st['term'].faces1, case['sigma_dist'])
        pa = torch.zeros_like(px)
        for t in range(T - 1, -1, -1):
            px, pa = _so_adjoint(case, xt[t], at[t], px, pa, dt)
        x, a = xt[0], at[0]
        ka = _k(case, x, x, a)
        kx = torch.cat([-_pull(_radial(case, _dist(x[s], x))[1] * (a[s] @ a.T), x[s], x)
                        for s in _rows(x.shape[0])]) / case['sigma'] ** 2
        return {'loss': e + e1 + 0.5 * (a * ka).sum(), 'dx0': px + kx, 'da0': pa + ka}
    # the network's training step from its bf16 weights and inputs, without the rounding of the activations
    m, n = st['model'], case['n']
    W = [w.double().requires_grad_() for w in m.Wb]
    b = [v.double().requires_grad_() for v in m.b]
    h = st['F'].double()
    for i in range(4):
        h = h @ W[i] + b[i]
        h = torch.relu(h) if i < 3 else h
    loss = ((h[:, :N_OUT] - st['target'].double()) ** 2).sum() / n
    return {'loss': loss.detach(), 'grads': list(torch.autograd.grad(loss, W + b)), 'weights': [None] * 4,
            'bias': [None] * 4}

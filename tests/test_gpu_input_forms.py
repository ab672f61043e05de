"""Forms of input that the entry points convert: lists, integer and CPU tensors, several widths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_data_term_takes_integer_target_vertices():
    """Vertices of whole numbers as an integer tensor: the values of the same vertices in float64."""
    import torch
    from base.kernelFunctions import Kernel
    from base.surfaceDistances import SurfaceDataTerm
    from base.syntheticShapes import icosphere
    v, f = icosphere(2)
    target = np.rint(8 * v)
    x = torch.from_numpy(8.3 * v).cuda()
    K = Kernel(name='gauss', sigma=3.0)
    ref = SurfaceDataTerm(f, target, f, K, nv=v.shape[0]).energy(x)
    for t in (torch.from_numpy(target.astype(np.int64)), torch.from_numpy(target.astype(np.int32)).cuda(),
              target.tolist()):
        assert torch.allclose(SurfaceDataTerm(f, t, f, K, nv=v.shape[0]).energy(x), ref, rtol=1e-12)


@pytest.mark.parametrize('n', [50, 9001])
def test_laplacian_sum_of_several_widths_and_columns(n, monkeypatch):
    """One origin serves every width and column group, and a host array's is averaged on the host; 2e-5 is the FP32
    tolerance of a kernel sum."""
    import torch
    import base._native as nat
    from base.kernelFunctions import Kernel
    r = np.random.default_rng(n)
    x, a = r.normal(size=(n, 3)), r.normal(size=(n, 4))
    K = Kernel(name='laplacian', sigma=[0.5, 0.8], order=2)
    calls = []
    centroid = nat.centroid
    monkeypatch.setattr(nat, 'centroid', lambda t: calls.append(type(t)) or centroid(t))
    K.pk_dtype = 'float32'
    out = K.applyK(x.tolist() if n == 50 else x, a)
    assert calls == ([] if n == 50 else [np.ndarray])
    K.pk_dtype = 'float64'
    ref = K.applyK(torch.from_numpy(x).cuda(), torch.from_numpy(a).cuda()).cpu().numpy()
    assert np.linalg.norm(out - ref) < 2e-5 * np.linalg.norm(ref)

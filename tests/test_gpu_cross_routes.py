"""Vector::cross and the bootstrap over the sides where their passes change
form, against numpy in FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = {torch.complex128: 1e-12, torch.complex64: 5e-6}


def _fields(shape, dtype, device, seed, count):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return [torch.complex(torch.randn(shape, generator=g, dtype=torch.float64),
                          torch.randn(shape, generator=g, dtype=torch.float64)).to(device, dtype)
            for _ in range(count)]


def _forward(f):
    f = np.fft.fftn(f)
    f[f.shape[0] // 2] = 0
    f[:, f.shape[1] // 2] = 0
    f[:, :, f.shape[2] // 2] = 0
    return f


def _cross(a, b):
    u, w = ([np.fft.ifftn(x) for x in v] for v in (a, b))
    return [_forward(u[(d + 1) % 3] * w[(d + 2) % 3] - u[(d + 2) % 3] * w[(d + 1) % 3])
            for d in range(3)]


def _host(v):
    return [x.to(torch.complex128).cpu().numpy() for x in v]


def _err(got, ref):
    n = np.linalg.norm(ref)
    return np.linalg.norm(got - ref) / n if n else np.linalg.norm(got)


# (nz, ny, nx): one and two points per side, the ends of the fused x pass (4,
# 1024) and beyond, planes of one CTA and just above, long y and z lines
@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("shape", [(1, 8, 8), (8, 1, 8), (8, 8, 1), (8, 8, 2), (2, 2, 4),
                                   (16, 16, 16), (4, 64, 64), (4, 128, 64), (2, 4, 1024),
                                   (2, 2, 2048), (512, 4, 8), (4, 1024, 8), (32, 128, 128)])
def test_cross_matches_numpy(sns, cuda, dtype, shape):
    a, b = _fields(shape, dtype, cuda, 1, 3), _fields(shape, dtype, cuda, 2, 3)
    keep = [x.clone() for x in a + b]
    got = sns.cross(a, b)
    for x, y in zip(a + b, keep):
        assert torch.equal(x, y)  # the operands are read only
    for g, r in zip(_host(got), _cross(_host(a), _host(b))):
        assert _err(g, r) < TOL[dtype]


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("shape", [(4, 8, 16), (32, 16, 64), (16, 128, 64)])
def test_bootstrap_matches_numpy(sns, cuda, dtype, shape):
    """V1 = V0 + dt (t - grad ilap(div t)), t = cross0 + nu laplacian(V0)."""
    nu, dt = 0.02, 3e-3
    k = [np.fft.fftfreq(n, 1 / n) for n in shape]
    for q, n in enumerate(shape):
        k[q][n // 2] = n // 2  # Scalar::freq: +n/2
    K = np.meshgrid(*k, indexing="ij")[::-1]
    k2 = sum(x * x for x in K)
    V = _fields(shape, dtype, cuda, 3, 3)
    w = sns.curl(V)
    st = sns.NSStepper(shape, nu, dt, dtype)
    st.bootstrap(V, w)
    got = st.state()
    st.close()
    v = _host(V)
    c = _cross(v, _host(w))
    t = [c[d] - nu * k2 * v[d] for d in range(3)]
    div = 1j * sum(K[d] * t[d] for d in range(3))
    p = np.where(k2 > 0, div / np.where(k2 > 0, -k2, 1), div)
    for d in range(3):
        assert _err(_host(got["cross0"])[d], c[d]) < TOL[dtype]
        assert _err(_host(got["V1"])[d], v[d] + dt * (t[d] - 1j * K[d] * p)) < TOL[dtype]

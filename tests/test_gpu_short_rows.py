"""Transforms along short x lines (staged through shared memory from 8 elements to
512 bytes) and passes over several fields (runs of tiles per field)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

U = {torch.complex128: 2.0 ** -53, torch.complex64: 2.0 ** -24}


def _field(shape, dtype, device, seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return torch.randn(shape, generator=g, dtype=torch.complex128).to(device, dtype)


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("nx", [4, 8, 16, 32, 64, 128])
@pytest.mark.parametrize("nz,ny", [(1, 1), (1, 2), (4, 8), (16, 64)])
def test_x_lines_match_torch(sns, cuda, dtype, nx, nz, ny):
    """Relative L2 error of a radix FFT: at most 2 log2(n) units (the reference's
    own error doubles that for complex128)."""
    f = _field((nz, ny, nx), dtype, cuda, nx + ny)
    N = sns._native
    prec = N.SNS_C128 if dtype == torch.complex128 else N.SNS_C64
    for sign, scale in ((-1, 1.0), (1, 0.25)):
        t = f.clone()
        N.call("sns_fft3d_axes", t.data_ptr(), nx, ny, nz, 1, sign, scale, prec,
               torch.cuda.current_stream().cuda_stream)
        d = f.to(torch.complex128)
        ref = scale * (torch.fft.fft(d) if sign < 0 else torch.fft.ifft(d, norm="forward"))
        err = torch.linalg.vector_norm(t.to(torch.complex128) - ref) / torch.linalg.vector_norm(ref)
        assert err < 4 * math.log2(nx) * U[dtype]


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("shape", [(1, 1, 16), (1, 1, 64), (2, 2, 8), (4, 64, 16), (32, 16, 64),
                                   (2, 2, 1024), (64, 64, 128)])
def test_several_fields_equal_one(sns, cuda, dtype, shape):
    """The tiles of five fields, whatever their order, are those of one field: the
    same bits, Nyquist zeroing and normalisation included."""
    fs = [_field(shape, dtype, cuda, i) for i in range(5)]
    many = [f.clone() for f in fs]
    sns.fft3d(many, -1, zero_nyquist=True)
    one = [sns.forward(f.clone()) for f in fs]
    for a, b in zip(many, one):
        assert torch.equal(a, b)
    sns.fft3d(many, 1, normalise=True)
    for a, b in zip(many, one):
        assert torch.equal(a, sns.inverse(b))

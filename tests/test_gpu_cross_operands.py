"""Operands of Vector::cross that its first pass cannot read in place."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(shape, dtype, device, offset):
    """Six contiguous fields whose first bytes lie `offset` bytes into buffers of
    their own."""
    g = torch.Generator(device="cpu").manual_seed(7)
    n = int(np.prod(shape)) * dtype.itemsize
    fields, ptrs, keep = [], [], []
    for _ in range(6):
        f = torch.randn(shape, generator=g, dtype=dtype).to(device)
        buf = torch.zeros(n + 16, dtype=torch.uint8, device=device)
        buf[offset:offset + n] = f.reshape(-1).view(torch.uint8)
        fields.append(f)
        keep.append(buf)
        ptrs.append(buf.data_ptr() + offset)
    return fields, ptrs, keep


# offset in bytes: whole elements that no TMA copy can start at, and (complex128,
# then complex64) half elements
@pytest.mark.parametrize("dtype,offset", [(torch.complex64, 8), (torch.complex128, 8),
                                          (torch.complex64, 4)])
@pytest.mark.parametrize("stages", ["0", "1"])
@pytest.mark.parametrize("shape", [(64, 128, 128), (16, 32, 32)])
def test_cross_of_unaligned_operands(sns, cuda, monkeypatch, dtype, offset, stages, shape):
    """Same bits as with aligned operands, whatever form the passes take."""
    monkeypatch.setenv("SNS_FFT_TMA", stages)
    N = sns._native
    fields, ptrs, keep = _operands(shape, dtype, cuda, offset)
    want = sns.cross(fields[:3], fields[3:])
    got = [torch.zeros_like(w) for w in want]
    nz, ny, nx = shape
    N.call("sns_cross", N.ptr3(ptrs[:3]), N.ptr3(ptrs[3:]), N.ptr3([x.data_ptr() for x in got]),
           nx, ny, nz, N.SNS_C64 if dtype == torch.complex64 else N.SNS_C128,
           torch.cuda.current_stream().cuda_stream)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    del keep

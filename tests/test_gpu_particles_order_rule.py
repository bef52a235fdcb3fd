"""Populations on both sides of the line from which moves are ordered."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


# (nz, ny, nx): fields of 170, 262 and 403 MB; the population is split into calls
# below the line, which move the particles as they are
@pytest.mark.parametrize("dtype,shape,n", [
    (torch.complex64, (192, 192, 192), 700_003),
    (torch.complex128, (176, 176, 176), 550_001),
    (torch.complex64, (64, 512, 512), 550_001),
    (torch.complex64, (4, 2048, 2048), 549_999),
])
def test_ordered_moves_equal_small_calls_bit_for_bit(sns, cuda, dtype, shape, n):
    g = torch.Generator(device=cuda).manual_seed(5)
    u = [torch.randn(shape, generator=g, device=cuda, dtype=torch.float64).to(dtype)
         for _ in range(3)]
    pos = torch.rand((n, 3), generator=g, device=cuda, dtype=torch.float64) * (2 * math.pi)
    pos[:4] = torch.tensor([[0.0, 0.0, 0.0], [2 * math.pi] * 3, [-0.5, 7.0, 3.0],
                            [3.0, -1e300, 1e300]], dtype=torch.float64, device=cuda)
    whole = sns.Tracers(pos.clone())
    parts = [sns.Tracers(p.clone()) for p in pos.split(1 << 17)]
    for _ in range(2):
        whole.move(u, 0.01)
        for p in parts:
            p.move(u, 0.01)
    bits = lambda x: x.view(torch.int64)  # noqa: E731  (infinities and NaN among them)
    assert torch.equal(bits(whole.pos), bits(torch.cat([p.pos for p in parts])))
    assert torch.equal(bits(whole.vel), bits(torch.cat([p.vel for p in parts])))

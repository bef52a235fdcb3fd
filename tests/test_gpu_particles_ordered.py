"""Large populations in fields beyond L2 are moved in another order
(sns_particles_move); the order must not show in the results."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


# (nz, ny, nx): z-major bands, fewer planes than bands, fewer rows than a band
@pytest.mark.parametrize("dtype,shape", [
    (torch.complex64, (128, 192, 240)),
    (torch.complex64, (4, 1024, 1296)),
    (torch.complex128, (2, 2, 1 << 20)),
])
def test_ordered_moves_equal_small_calls_bit_for_bit(sns, cuda, dtype, shape):
    """(1 << 17) + 77 particles in one call take the ordered route, the same
    particles in calls of at most 1 << 16 the direct one.  Positions at both
    ends of the box, on its upper face and outside it are among them."""
    g = torch.Generator(device=cuda).manual_seed(5)
    u = [torch.randn(shape, generator=g, device=cuda, dtype=torch.float64).to(dtype)
         for _ in range(3)]
    n = (1 << 17) + 77
    assert 3 * u[0].numel() * u[0].element_size() > 126e6  # the ordered route's condition
    assert n * 64 >= u[0].numel()
    pos = torch.rand((n, 3), generator=g, device=cuda, dtype=torch.float64) * (2 * math.pi)
    pos[:4] = torch.tensor([[0.0, 0.0, 0.0], [2 * math.pi] * 3, [-0.5, 7.0, 3.0],
                            [3.0, -1e300, 1e300]], dtype=torch.float64, device=cuda)
    whole = sns.Tracers(pos.clone())
    parts = [sns.Tracers(p.clone()) for p in pos.split(1 << 16)]
    for _ in range(2):
        whole.move(u, 0.01)
        for p in parts:
            p.move(u, 0.01)
    # the bits: positions far outside the box extrapolate to infinities and NaN
    bits = lambda x: x.view(torch.int64)  # noqa: E731
    assert torch.equal(bits(whole.pos), bits(torch.cat([p.pos for p in parts])))
    assert torch.equal(bits(whole.vel), bits(torch.cat([p.vel for p in parts])))

"""Steppers of boxes whose planes fit a CTA (plane pass + carrying update pass,
batched graphs) against the five separate passes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fourier_of_real(shape, dtype, device, seed):
    """Fourier transforms of real random fields, Nyquist planes zero."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    out = []
    for _ in range(3):
        f = torch.fft.fftn(torch.randn(shape, generator=g, dtype=torch.float64).to(device))
        f[shape[0] // 2] = 0
        f[:, shape[1] // 2] = 0
        f[:, :, shape[2] // 2] = 0
        out.append(f.to(dtype))
    return out


# the smallest planes, the largest that fit (complex64 / complex128), uneven
# ones, lines of every elements-per-thread choice along z (16, 64, 128, 512)
@pytest.mark.parametrize("dtype,shape,real", [
    (torch.complex64, (16, 16, 16), False),
    (torch.complex64, (4, 16, 32), False),
    (torch.complex64, (32, 32, 32), False),
    (torch.complex64, (32, 32, 32), True),
    (torch.complex64, (64, 64, 64), False),
    (torch.complex64, (16, 64, 128), True),
    (torch.complex64, (128, 256, 16), False),
    (torch.complex64, (8, 16, 256), False),
    (torch.complex64, (512, 32, 16), False),
    (torch.complex128, (16, 16, 16), False),
    (torch.complex128, (32, 32, 64), False),
    (torch.complex128, (64, 32, 128), True),
    (torch.complex128, (64, 128, 16), False),
])
def test_plane_plan_matches_separate_passes(sns, cuda, monkeypatch, dtype, shape, real):
    """Both plans do the step of ns.cpp:167-217; line FFTs with other radix
    orders differ by rounding, a few units a step: 1 + 11 + 3 steps (an eager
    one, one batched graph and single replays, a new state) stay within 50
    rounding units."""
    V = _fourier_of_real(shape, dtype, cuda, 3)
    V2 = _fourier_of_real(shape, dtype, cuda, 4)
    scale = 1.0 / (shape[0] * shape[1] * shape[2]) ** 0.5
    out, stats = {}, {}
    for mode in ("0", "1"):
        monkeypatch.setenv("SNS_PLANE", mode)
        st = sns.NSStepper(shape, 1 / 100, 1e-4, dtype, real=real)
        assert ("xy=plane" in st.describe()) == (mode == "1"), st.describe()
        assert st.launches_per_step() == (2 if mode == "1" else 5)
        st.set_state([scale * v for v in V], [scale * v for v in V2])
        st.step(1)
        st.step(11)
        mid = st.state()
        stats[mode] = st.stats()
        st.set_state([scale * v for v in V2], [scale * v for v in V])
        st.step(3)
        out[mode] = mid["V1"] + mid["cross0"] + st.state()["V1"] + st.state()["omega1"]
        st.close()
    eps = 1.2e-7 if dtype == torch.complex64 else 2.3e-16
    for a, b in zip(out["1"], out["0"]):
        err = (torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b)).item()
        assert err < 50 * eps, err
    for k in ("energy", "enstrophy"):
        assert abs(stats["1"][k] / stats["0"][k] - 1) < 100 * eps, k


def test_planes_that_do_not_fit_keep_the_separate_passes(sns, cuda):
    for dtype, shape in ((torch.complex64, (16, 128, 64)), (torch.complex128, (16, 64, 64)),
                         (torch.complex64, (64, 8, 64)), (torch.complex64, (16, 512, 16))):
        st = sns.NSStepper(shape, 1 / 100, 1e-4, dtype)
        assert "xy=separate" in st.describe(), st.describe()
        st.close()

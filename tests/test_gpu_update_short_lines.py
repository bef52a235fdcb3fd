"""Update-pass tiles whose width does not divide their thread count."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one thread per z line (nz <= 16) and a tile in two halves: 3 W / 2 threads
@pytest.mark.parametrize("dtype,nx,wide", [(torch.complex128, 256, "256"),
                                           (torch.complex64, 512, "512")])
@pytest.mark.parametrize("nz", [4, 8, 16])
def test_wide_tile_of_short_lines_bit_for_bit(sns, cuda, dtype, nx, wide, nz, monkeypatch):
    """Three steps (the first from a Fourier history, the others from one before
    its z-forward) give the same bits as narrow tiles."""
    shape = (nz, 8, nx)
    g = torch.Generator(device="cpu").manual_seed(5)
    f = [torch.randn(shape, generator=g, dtype=torch.complex128).to(cuda, dtype) for _ in range(6)]
    out, stats = {}, {}
    for mode in ("4", wide):
        monkeypatch.setenv("SNS_Z_W", mode)
        st = sns.NSStepper(shape, 1 / 400, 5e-4, dtype)
        assert "zW=%s" % mode in st.describe(), st.describe()
        st.set_state(f[:3], f[3:])
        st.step(3)
        assert sns._native.lib().sns_ns_check(st.h) == 0
        q = st.state()
        out[mode] = q["V1"] + q["cross0"]
        stats[mode] = st.stats()
        st.close()
    for a, b in zip(out[wide], out["4"]):
        assert torch.equal(a, b)
    for k in stats["4"]:  # partials summed in another order
        assert abs(stats[wide][k] - stats["4"][k]) <= 1e-12 * abs(stats["4"][k])

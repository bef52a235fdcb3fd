"""What the tuners time (their log)."""
import re

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_stepper_tuner_times_the_default_and_small_ctas(sns, cuda, monkeypatch, capfd, dtype):
    """Every stage lists the plan it would replace first, and the y passes' stage
    the thread cap of the default tile."""
    monkeypatch.setenv("SNS_TUNE_LOG", "1")
    monkeypatch.setenv("SNS_PLANE", "0")
    sns.NSStepper((8, 64, 128), 0.01, 1e-4, dtype, tune=True).close()
    log = capfd.readouterr().err
    y = re.findall(r"ns_tune passes=0xa cand=(\d+) .*lineW=(\d+) lineT=(\d+)", log)
    assert ("0", "0", "0") in y, y[:4]
    assert any(t == "64" for _, _, t in y)
    # and the whole step of what was chosen is compared with the default's
    assert re.findall(r"ns_tune passes=0x1f cand=0 .*lineW=(\d+) lineT=(\d+)", log)[0] == ("0", "0")
    x = re.findall(r"ns_tune passes=0x4 cand=0 .* xG=(\S+) ", log)
    z = re.findall(r"ns_tune passes=0x10 cand=0 .* zW=(\S+) ", log)
    monkeypatch.delenv("SNS_TUNE_LOG")
    st = sns.NSStepper((8, 64, 128), 0.01, 1e-4, dtype)
    d = st.describe()
    st.close()
    assert f"xG={x[0]} " in d + " " and f"zW={z[0]} " in d, (x, z, d)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_transform_tuner_times_the_default_and_small_ctas(sns, cuda, monkeypatch, capfd, dtype):
    monkeypatch.setenv("SNS_TUNE_LOG", "1")
    sns.fft3d_tune((8, 64, 128), dtype, nfields=2, device=cuda)
    log = capfd.readouterr().err
    for axis in (0, 1, 2):
        seen = re.findall(rf"fft3d_tune axis={axis} W=(\d+) T=(\d+) tma=(\d)", log)
        w = "16" if axis == 0 or dtype == torch.complex64 else "8"
        assert (w, "64", "0") in seen  # the default tile

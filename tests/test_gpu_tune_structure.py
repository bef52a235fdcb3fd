"""Tuned plans of steppers of one box that run different pass structures."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,order", [((64, 32, 16), ("0", "1")), ((64, 16, 32), ("1", "0"))])
def test_a_tuned_plan_keeps_the_steppers_structure(sns, cuda, monkeypatch, shape, order):
    for mode in order + order:
        monkeypatch.setenv("SNS_PLANE", mode)
        st = sns.NSStepper(shape, 0.01, 1e-4, torch.complex64, tune=True)
        assert ("xy=plane" in st.describe()) == (mode == "1"), (mode, st.describe())
        assert st.launches_per_step() == (2 if mode == "1" else 5)
        f = [torch.zeros(shape, dtype=torch.complex64, device=cuda) for _ in range(6)]
        st.set_state(f[:3], f[3:])
        st.step(3)
        assert sns._native.lib().sns_ns_check(st.h) == 0
        st.close()

"""Boxes on both sides of the line from which the plane pass is chosen."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,shape,real,plane", [
    (torch.complex64, (32, 64, 64), False, False),
    (torch.complex64, (64, 64, 64), False, True),
    (torch.complex64, (8, 256, 16), False, False),
    (torch.complex64, (16, 256, 16), False, True),
    (torch.complex64, (64, 16, 512), True, False),
    (torch.complex64, (128, 16, 512), True, True),
    (torch.complex64, (4, 32, 64), False, True),
    (torch.complex128, (8, 32, 64), False, False),
    (torch.complex128, (16, 32, 64), False, True),
    (torch.complex128, (16, 64, 64), True, False),
    (torch.complex128, (32, 64, 64), True, True),
    (torch.complex128, (4, 32, 32), False, True),
])
def test_few_large_planes_take_the_separate_passes(sns, cuda, dtype, shape, real, plane):
    st = sns.NSStepper(shape, 0.01, 1e-4, dtype, real=real)
    assert ("xy=plane" in st.describe()) == plane, st.describe()
    assert st.launches_per_step() == (2 if plane else 5)
    st.close()

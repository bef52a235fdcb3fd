"""Fields that kernels of the device cannot read: only a copy may touch them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_host_fields_end_in_a_copy_or_an_error(sns, cuda):
    """Pageable host memory given as a state, as operands and as read-back goes to
    the copy engine, which takes or refuses it on the host; the device and the
    stepper stay usable."""
    N = sns._native
    shape, dtype = (16, 16, 32), torch.complex64
    nz, ny, nx = shape
    host = [torch.randn(shape, dtype=dtype) for _ in range(6)]
    dev = [x.to(cuda) for x in host]
    hp, dp = [x.data_ptr() for x in host], [x.data_ptr() for x in dev]
    st = sns.NSStepper(shape, 0.01, 1e-4, dtype)
    ens = sns.NSEnsemble([shape], [0.01], 1e-4, dtype, tune=False)
    out = [torch.zeros_like(x) for x in dev]
    s = torch.cuda.current_stream().cuda_stream
    taken = []
    for a, b in ((hp[:3], dp[3:]), (dp[:3], hp[3:])):
        taken.append(N.lib().sns_ns_set_state(st.h, N.ptr3(a), N.ptr3(b)))
        taken.append(N.lib().sns_ens_set_state(ens.h, 0, N.ptr3(a), N.ptr3(b)))
        taken.append(N.lib().sns_cross(N.ptr3(a), N.ptr3(b),
                                       N.ptr3([x.data_ptr() for x in out[:3]]), nx, ny, nz,
                                       st.prec, s))
        torch.cuda.synchronize()
    st.set_state(dev[:3], dev[3:])
    ens.set_state(0, dev[:3], dev[3:])
    st.step(2)
    ens.step(2)
    back = [torch.zeros(shape, dtype=dtype) for _ in range(6)]
    bp = [x.data_ptr() for x in back]
    w = [x.data_ptr() for x in out[:3]]
    for rc in (N.lib().sns_ns_get_state(st.h, N.ptr3(bp[:3]), N.ptr3(w), N.ptr3(bp[3:])),
               N.lib().sns_ens_get_state(ens.h, 0, N.ptr3(bp[:3]), N.ptr3(w), N.ptr3(bp[3:]))):
        taken.append(rc)
        torch.cuda.synchronize()
        if rc == N.SNS_OK:
            q = st.state()
            for x, y in zip(back, q["V1"] + q["cross0"]):
                assert torch.equal(x, y.cpu())
    assert all(rc in (N.SNS_OK, N.SNS_ERR_CUDA) for rc in taken), taken
    ref = sns.NSStepper(shape, 0.01, 1e-4, dtype)
    ref.set_state(dev[:3], dev[3:])
    ref.step(3)
    st.step(1)
    ens.step(1)
    for got in (st.state(), ens.state(0)):
        for x, y in zip(got["V1"], ref.state()["V1"]):
            assert (torch.linalg.vector_norm(x - y) / torch.linalg.vector_norm(y)).item() < 1e-5
    for q in (st, ens, ref):
        q.close()

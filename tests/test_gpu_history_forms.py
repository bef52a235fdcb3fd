"""The stepper's history between calls: steps leave it before its z-forward, and
closures, cutoffs, read-backs and new states take it from there."""
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = {torch.complex64: 1.2e-7, torch.complex128: 2.3e-16}


def _state(shape, dtype, device, seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    out = []
    for _ in range(6):
        f = torch.fft.fftn(torch.randn(shape, generator=g, dtype=torch.float64).to(device))
        f[shape[0] // 2] = 0
        f[:, shape[1] // 2] = 0
        f[:, :, shape[2] // 2] = 0
        out.append((f / f.numel() ** 0.5).to(dtype))
    return out[:3], out[3:]


def _close(got, want, dtype):
    """A history set as Fourier fields joins the step after its transform, one left
    by a step before it: a few rounding units a step."""
    for k in ("V1", "cross0"):
        for a, b in zip(got[k], want[k]):
            err = (torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b)).item()
            assert err < 100 * EPS[dtype], (k, err)


@pytest.mark.parametrize("dtype,shape", [(torch.complex64, (32, 32, 32)),
                                         (torch.complex128, (16, 32, 32)),
                                         (torch.complex64, (16, 128, 64))])
@pytest.mark.parametrize("before", [1, 2, 10])
def test_closures_and_cutoffs_after_plain_steps(sns, cuda, dtype, shape, before):
    """At every change a second stepper is set to the state read back from the
    first, so its history starts as Fourier fields."""
    N = sns._native
    a = sns.NSStepper(shape, 0.01, 1e-4, dtype)
    a.set_state(*_state(shape, dtype, cuda, 1))
    changes = [(N.SNS_CLOSURE_SMAGORINSKY, 1e-3, 0.0, 2), (N.SNS_CLOSURE_NONE, 0.0, 0.0, before),
               (N.SNS_CLOSURE_NONE, 0.0, 9.0, before), (N.SNS_CLOSURE_NONE, 0.0, 5.0, 1),
               (N.SNS_CLOSURE_SMAGORINSKY, 1e-3, 6.0, 1), (N.SNS_CLOSURE_NONE, 0.0, 0.0, 3)]
    a.step(before)
    for model, cs, kc, steps in changes:
        q = a.state()
        b = sns.NSStepper(shape, 0.01, 1e-4, dtype)
        b.set_state(q["V1"], q["cross0"])
        for st in (a, b):
            st.set_closure(model, cs, kc=kc)
            st.step(steps)
        got, want = a.state(), b.state()
        _close(got, want, dtype)
        if kc:
            k = [torch.fft.fftfreq(n, 1 / n, device=cuda) for n in shape]
            k2 = k[0][:, None, None] ** 2 + k[1][:, None] ** 2 + k[2] ** 2
            assert all(not x[k2 > kc * kc].any() for x in got["V1"] + got["cross0"])
        b.close()
    a.close()


@pytest.mark.parametrize("dtype,offset", [(torch.complex64, 4), (torch.complex128, 8)])
@pytest.mark.parametrize("steps", [0, 1, 2])
def test_state_read_into_unaligned_memory(sns, cuda, dtype, offset, steps):
    N = sns._native
    shape = (16, 32, 32)
    V, c = _state(shape, dtype, cuda, 2)
    st = sns.NSStepper(shape, 0.01, 1e-4, dtype)
    ens = sns.NSEnsemble([shape], [0.01], 1e-4, dtype, tune=False)
    st.set_state(V, c)
    ens.set_state(0, V, c)
    st.step(steps)
    ens.step(steps)
    n = V[0].numel() * dtype.itemsize
    for read, want in ((lambda v, x: N.call("sns_ns_get_state", st.h, v, None, x), st.state()),
                       (lambda v, x: N.call("sns_ens_get_state", ens.h, 0, v, None, x),
                        ens.state(0))):
        buf = [torch.zeros(n + 16, dtype=torch.uint8, device=cuda) for _ in range(6)]
        p = [x.data_ptr() + offset for x in buf]
        read(N.ptr3(p[:3]), N.ptr3(p[3:]))
        for x, w in zip(buf, want["V1"] + want["cross0"]):
            got = x[offset:offset + n].clone().view(dtype).reshape(shape)
            assert torch.equal(got, w)
            assert not x[:offset].any() and not x[offset + n:].any()
    st.close()
    ens.close()


def test_boxes_set_between_steps_in_mixed_modes(sns, cuda):
    shapes, nus, dtype = [(32, 32, 32), (16, 32, 64), (32, 32, 32)], [0.01, 0.02, 0.03], torch.complex64
    ens = sns.NSEnsemble(shapes, nus, 1e-4, dtype, tune=False)
    one = [sns.NSStepper(s, nu, 1e-4, dtype) for s, nu in zip(shapes, nus)]

    def put(i, seed):
        V, c = _state(shapes[i], dtype, cuda, seed)
        ens.set_state(i, V, c)
        one[i].set_state(V, c)

    for i in range(3):
        put(i, i)
    modes = [sns.ENS_GRAPH, sns.ENS_EAGER, sns.ENS_SEQUENTIAL]
    for turn, (n, mode, box) in enumerate([(1, 0, 1), (2, 1, 2), (1, 2, 0), (3, 0, 1), (1, 1, 0),
                                           (2, 2, 2), (1, 0, None)]):
        ens.step(n, modes[mode])
        for i, st in enumerate(one):
            st.step(n)
            _close(ens.state(i), st.state(), dtype)
        if box is not None:
            put(box, 10 + turn)
    ens.close()
    for st in one:
        st.close()

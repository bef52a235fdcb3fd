"""Read-back of a real-field stepper's history."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(32, 32, 32), (16, 128, 64)])
def test_history_is_read_without_a_synchronisation(sns, cuda, shape):
    """A read of V1 and cross0 after steps is queued on the stepper's stream: it
    returns while the stream still runs what was queued before.  Reading leaves
    the following steps as they are."""
    N = sns._native
    g = torch.Generator(device="cpu").manual_seed(3)
    f = [torch.fft.fftn(torch.randn(shape, generator=g)).to(cuda) / 64 for _ in range(6)]
    a, b = (sns.NSStepper(shape, 0.01, 1e-4, torch.complex64, real=True) for _ in range(2))
    for q in (a, b):
        q.set_state(f[:3], f[3:])
    out = [torch.zeros_like(x) for x in f]
    # (the first launch of a kernel may load it)
    warm = sns.NSStepper(shape, 0.01, 1e-4, torch.complex64, real=True)
    warm.set_state(f[:3], f[3:])
    warm.step(3)
    N.call("sns_ns_get_state", warm.h, warm._vec(out[:3]), None, warm._vec(out[3:]))
    for n in (1, 2, 9):
        for q in (a, b):
            q.step(n)
        torch.cuda.synchronize()
        torch.cuda._sleep(500_000_000)  # about a quarter of a second
        done = torch.cuda.Event()
        done.record()
        N.call("sns_ns_get_state", b.h, b._vec(out[:3]), None, b._vec(out[3:]))
        assert not done.query()
    a.step(1)
    b.step(1)
    want = a.state()
    N.call("sns_ns_get_state", b.h, b._vec(out[:3]), None, b._vec(out[3:]))
    for x, y in zip(out, want["V1"] + want["cross0"]):
        err = (torch.linalg.vector_norm(x - y) / torch.linalg.vector_norm(y)).item()
        assert err < 100 * 1.2e-7, err
    warm.close()
    a.close()
    b.close()

"""Steps captured by the caller into a CUDA graph of its own and replayed."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _state(shape, dtype, device, seed):
    """Fourier transforms of real random fields, Nyquist planes zero."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    out = []
    for _ in range(6):
        f = torch.fft.fftn(torch.randn(shape, generator=g, dtype=torch.float64).to(device))
        f[shape[0] // 2] = 0
        f[:, shape[1] // 2] = 0
        f[:, :, shape[2] // 2] = 0
        out.append((f / f.numel() ** 0.5).to(dtype))
    return out[:3], out[3:]


def _close(got, want, eps):
    """Line FFTs of other orders, and the history's z-forward on its own instead
    of joined with the new product, differ by a few rounding units a step."""
    for k in ("V1", "omega1", "cross0"):
        for a, b in zip(got[k], want[k]):
            err = (torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b)).item()
            assert err < 100 * eps, (k, err)


@pytest.mark.parametrize("dtype,shape,real", [
    (torch.complex64, (32, 32, 32), False),   # plane pass, carried K1
    (torch.complex64, (32, 32, 32), True),
    (torch.complex64, (16, 128, 64), False),  # five passes
    (torch.complex128, (16, 64, 64), False),
])
@pytest.mark.parametrize("n,before", [(1, 0), (1, 2), (3, 1), (2, 9)])
def test_replayed_steps_advance_the_state(sns, cuda, dtype, shape, real, n, before):
    eps = 1.2e-7 if dtype == torch.complex64 else 2.3e-16
    a, b = _state(shape, dtype, cuda, 1), _state(shape, dtype, cuda, 2)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        warm = sns.NSStepper(shape, 0.01, 1e-4, dtype, real=real)  # tables and attributes
        warm.set_state(*a)
        warm.step(20)
        ref = sns.NSStepper(shape, 0.01, 1e-4, dtype, real=real)
        st = sns.NSStepper(shape, 0.01, 1e-4, dtype, real=real)
        for q in (ref, st):
            q.set_state(*a)
            q.step(before)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            st.step(n)
        _close(st.state(), ref.state(), eps)  # nothing of the capture has run
        for _ in range(3):
            g.replay()
        ref.step(3 * n)
        _close(st.state(), ref.state(), eps)
        # direct steps between replays
        st.step(1)
        g.replay()
        ref.step(1 + n)
        _close(st.state(), ref.state(), eps)
        # a new state, then replays
        for q in (ref, st):
            q.set_state(*b)
        g.replay()
        g.replay()
        ref.step(2 * n)
        _close(st.state(), ref.state(), eps)
        torch.cuda.synchronize()
        del g
        for q in (warm, ref, st):
            q.close()


def test_state_set_and_read_inside_a_capture(sns, cuda):
    shape, dtype = (32, 32, 32), torch.complex64
    a, b = _state(shape, dtype, cuda, 1), _state(shape, dtype, cuda, 2)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        ref = sns.NSStepper(shape, 0.01, 1e-4, dtype)
        st = sns.NSStepper(shape, 0.01, 1e-4, dtype)
        for q in (ref, st):
            q.set_state(*a)
            q.step(3)
            q.state()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            st.set_state(*b)
            st.step(2)
            out = st.state()
        st.step(1)  # goes on from the state before the capture
        ref.step(1)
        _close(st.state(), ref.state(), 1.2e-7)
        for _ in range(2):
            g.replay()
            ref.set_state(*b)
            ref.step(2)
            _close(out, ref.state(), 1.2e-7)
        torch.cuda.synchronize()
        del g
        ref.close()
        st.close()


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("n,before", [(1, 0), (1, 1), (2, 3)])
def test_replayed_ensemble_steps_advance_the_state(sns, cuda, mode, n, before):
    shapes, dtype, eps = [(32, 32, 32), (16, 32, 64)], torch.complex64, 1.2e-7
    a = [_state(sh, dtype, cuda, 1 + i) for i, sh in enumerate(shapes)]
    b = [_state(sh, dtype, cuda, 5 + i) for i, sh in enumerate(shapes)]
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        ref, st = (sns.NSEnsemble(shapes, [0.01, 0.02], 1e-4, dtype, tune=False)
                   for _ in range(2))

        def check():
            for i in range(2):
                _close(st.state(i), ref.state(i), eps)

        for q in (ref, st):
            for i in range(2):
                q.set_state(i, *a[i])
            q.step(before + 2, mode)  # both places of the history have been used
            for i in range(2):
                q.set_state(i, *a[i])
            q.step(before, mode)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            st.step(n, mode)
        check()
        for _ in range(3):
            g.replay()
        ref.step(3 * n, mode)
        check()
        st.step(1, mode)
        g.replay()
        ref.step(1 + n, mode)
        check()
        for q in (ref, st):
            q.set_state(1, *b[1])
        g.replay()
        g.replay()
        ref.step(2 * n, mode)
        check()
        torch.cuda.synchronize()
        del g
        ref.close()
        st.close()


@pytest.mark.parametrize("ensemble", [False, True])
@pytest.mark.parametrize("n", [1, 2])
def test_reads_still_queued_when_a_capture_begins(sns, cuda, ensemble, n):
    """A read-back that waits in the stream when the first captured call moves the
    history to its place for replays reads it where it was."""
    shape, dtype = (32, 32, 32), torch.complex64
    a = _state(shape, dtype, cuda, 1)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    N = sns._native
    with torch.cuda.stream(s):
        if ensemble:
            ref, st = (sns.NSEnsemble([shape], [0.01], 1e-4, dtype, tune=False) for _ in range(2))
            read = lambda q: q.state(0)  # noqa: E731
        else:
            ref, st = (sns.NSStepper(shape, 0.01, 1e-4, dtype) for _ in range(2))
            read = lambda q: q.state()  # noqa: E731
        for q in (ref, st):
            q.set_state(0, *a) if ensemble else q.set_state(*a)
            q.step(2)  # kernels loaded, graphs captured
            read(q)
            q.set_state(0, *a) if ensemble else q.set_state(*a)
            q.step(n)
        want = read(ref)
        torch.cuda.synchronize()
        torch.cuda._sleep(200_000_000)  # about a tenth of a second
        got = read(st)
        g = torch.cuda.CUDAGraph()
        g.capture_begin()
        st.step(1)
        g.capture_end()
        torch.cuda.synchronize()
        for k in ("V1", "omega1", "cross0"):
            for x, y in zip(got[k], want[k]):
                assert torch.equal(x, y), k
        g.replay()
        ref.step(1)
        _close(read(st), read(ref), 1.2e-7)
        torch.cuda.synchronize()
        del g
        ref.close()
        st.close()

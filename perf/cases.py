"""Measured workloads of the framework, through its public entry points.

A case is a dict of plain values.  ``prepare`` makes what a program has in hand
before the call (fields, plans, steppers, models) from a seed, ``run`` is one
pass as such a program would call it, ``work`` the bytes and operations of a
pass that no implementation can avoid, ``exact`` the outputs in 64 bits from
plain torch.

Kinds and what they stand for:

* ``ns``: a segment of a Navier-Stokes run (exec/ns.cpp): the state is set, some
  steps are taken and the state is read back.  ``bootstrap`` starts from a
  velocity and its vorticity as ns.cpp does and reads the divergence monitor
  after every step.
* ``fft``: forward + inverse 3D transforms (exec/fft.cpp).
* ``poisson``: an in-place spectral Poisson solve (forward, inverse Laplacian,
  inverse).
* ``cross``: Vector::cross of two Fourier vectors, the nonlinear term of a
  program written against the field API.
* ``project``: the pressure projection of such a program from single operators.
* ``ens``: a segment of a batched ensemble of uneven boxes.
* ``les``: a segment of a coarse run with an eddy-viscosity closure.
* ``mlp``: validation and one gradient of the closure's model on filtered-DNS
  samples.
* ``tracers``: a population of particles moved through a velocity snapshot.

Fields have shape (nz, ny, nx).
"""
import math

import numpy as np
import torch

import spectral_upcxx_b200 as S
from spectral_upcxx_b200 import _native
from spectral_upcxx_b200 import closure

DEV = "cuda"
CLOSURES = {"none": _native.SNS_CLOSURE_NONE, "smagorinsky": _native.SNS_CLOSURE_SMAGORINSKY,
            "mlp": _native.SNS_CLOSURE_MLP}


def listed():
    return [
        # the headline benchmark: 256^3 DNS in single precision, tuned plan
        {"name": "ns_256_c64_tuned", "kind": "ns", "nx": 256, "ny": 256, "nz": 256, "dtype": "c64",
         "real": False, "tune": True, "steps": 20, "bootstrap": False},
        # the same box as exec/ns.cpp runs it: double precision from the
        # initial condition on, the divergence monitor read every step
        {"name": "ns_256_c128_monitored", "kind": "ns", "nx": 256, "ny": 256, "nz": 256,
         "dtype": "c128", "real": False, "tune": False, "steps": 10, "bootstrap": True},
        # a real velocity on the half spectrum, the constructor's default plan
        {"name": "ns_256_c64_real", "kind": "ns", "nx": 256, "ny": 256, "nz": 256, "dtype": "c64",
         "real": True, "tune": False, "steps": 20, "bootstrap": False},
        # the smallest boxes: a step is a few launches
        {"name": "ns_32_c64", "kind": "ns", "nx": 32, "ny": 32, "nz": 32, "dtype": "c64",
         "real": False, "tune": False, "steps": 40, "bootstrap": False},
        # the transform benchmark (exec/fft.cpp), tuned plan
        {"name": "fft_256_c64_tuned", "kind": "fft", "nx": 256, "ny": 256, "nz": 256,
         "dtype": "c64", "fields": 1, "tune": True},
        # three double-precision fields of uneven sides, default plan
        {"name": "poisson_16x256x512_c128", "kind": "poisson", "nx": 16, "ny": 256, "nz": 512,
         "dtype": "c128", "fields": 3, "tune": False},
        # the nonlinear term through the field API
        {"name": "cross_128_c128", "kind": "cross", "nx": 128, "ny": 128, "nz": 128,
         "dtype": "c128"},
        # eager operators on an odd grid (they take any size)
        {"name": "project_150x97x81_c64", "kind": "project", "nx": 150, "ny": 97, "nz": 81,
         "dtype": "c64"},
        # the ensemble benchmark: 64 boxes of three sizes, the default (tuned) plan
        {"name": "ens_64boxes_c64", "kind": "ens", "n32": 32, "n64": 24, "n128": 8,
         "dtype": "c64", "tune": True, "steps": 20},
        # the coarse run with the learned closure
        {"name": "les_64_mlp_c64", "kind": "les", "n": 64, "model": "mlp", "dtype": "c64",
         "steps": 20},
        # one minibatch of the closure's training and a validation pass
        {"name": "mlp_300001", "kind": "mlp", "rows": 300001, "batch": 262144},
        # tracers in a DNS snapshot
        {"name": "tracers_1M_256_c64", "kind": "tracers", "n": 256, "particles": 1000003,
         "dtype": "c64", "moves": 2},
    ]


# --------------------------------------------------------------------- drawing
def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pow2(rng, lo, hi):
    return 1 << rng.randint(lo.bit_length() - 1, hi.bit_length() - 1)


def _box(rng, lo, hi, most):
    """Three power-of-two sides in [lo, hi] of at most `most` points."""
    while True:
        d = [_pow2(rng, lo, hi) for _ in range(3)]
        if d[0] * d[1] * d[2] <= most:
            return d


def draw(rng):
    """One more case: small and large, cubic and uneven boxes of every kind."""
    kind = rng.choice(["ns", "ns", "ns", "fft", "fft", "poisson", "cross", "project", "ens", "les",
                       "mlp", "tracers"])
    dtype = rng.choice(["c64", "c64", "c128"])
    half = 2 if dtype == "c128" else 1
    if kind == "ns":
        nx, ny, nz = _box(rng, 32, 256, (1 << 24) // half)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "dtype": dtype,
                "real": rng.random() < 0.3, "tune": rng.random() < 0.25,
                "steps": rng.randint(3, 20), "bootstrap": rng.random() < 0.3}
    if kind in ("fft", "poisson"):
        nx, ny, nz = _box(rng, 16, 512, (1 << 24) // half)
        most = max(1, min(6, (1 << 25) // half // (nx * ny * nz)))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "dtype": dtype,
                "fields": rng.randint(1, most), "tune": rng.random() < 0.25}
    if kind == "cross":
        nx, ny, nz = _box(rng, 16, 256, (1 << 24) // half)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "dtype": dtype}
    if kind == "project":
        nx, ny, nz = (_log_uniform(rng, 9, 256) for _ in range(3))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "dtype": dtype}
    if kind == "ens":
        return {"kind": kind, "n32": rng.randint(1, 32), "n64": rng.randint(0, 12),
                "n128": rng.randint(0, 4), "dtype": dtype, "tune": rng.random() < 0.5,
                "steps": rng.randint(3, 10)}
    if kind == "les":
        return {"kind": kind, "n": rng.choice([32, 64, 128]),
                "model": rng.choice(["mlp", "smagorinsky"]), "dtype": dtype,
                "steps": rng.randint(3, 20)}
    if kind == "mlp":
        rows = _log_uniform(rng, 1000, 2000000)
        return {"kind": kind, "rows": rows, "batch": rng.randint(max(1, rows // 4), rows)}
    return {"kind": "tracers", "n": _pow2(rng, 32, 256),
            "particles": _log_uniform(rng, 1000, 2000000), "dtype": dtype,
            "moves": rng.randint(1, 4)}


# --------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _cdtype(case):
    return torch.complex64 if case["dtype"] == "c64" else torch.complex128


def _k1(n):
    """Scalar::freq: i for i <= n/2, else i - n."""
    i = torch.arange(n, device=DEV, dtype=torch.float64)
    return torch.where(i <= n // 2, i, i - n)


def _k(shape):
    nz, ny, nx = shape
    return _k1(nx)[None, None, :], _k1(ny)[None, :, None], _k1(nz)[:, None, None]


def _k2(shape):
    kx, ky, kz = _k(shape)
    return kx * kx + ky * ky + kz * kz


def _zero_nyquist(f):
    nz, ny, nx = f.shape
    f[nz // 2, :, :] = 0
    f[:, ny // 2, :] = 0
    f[:, :, nx // 2] = 0
    return f


def _forward(f):
    return _zero_nyquist(torch.fft.fftn(f))


def _ik(shape, d):
    return 1j * _k(shape)[d]


def _curl(v):
    ix, iy, iz = (_ik(v[0].shape, d) for d in range(3))
    return [iy * v[2] - iz * v[1], iz * v[0] - ix * v[2], ix * v[1] - iy * v[0]]


def _crossed(a, b):
    return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]


def _velocity(shape, g):
    """Fourier transform of a random solenoidal real velocity of unit rms with
    E(k) ~ k^4 exp(-2 (k/4)^2), Nyquist planes zero (complex128)."""
    k2 = _k2(shape)
    kmag = torch.sqrt(k2)
    safe = torch.where(k2 > 0, k2, torch.ones_like(k2))
    amp = torch.sqrt(kmag ** 4 * torch.exp(-2.0 * (kmag / 4.0) ** 2) / safe)
    v = []
    for _ in range(3):
        u = torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)
        v.append(_zero_nyquist(torch.fft.fftn(u)) * amp)
    k = _k(shape)
    div = (k[0] * v[0] + k[1] * v[1] + k[2] * v[2]) / safe
    v = [v[d] - k[d] * div for d in range(3)]
    n = shape[0] * shape[1] * shape[2]
    rms = math.sqrt(sum(float(x.abs().square().sum()) for x in v) / 3) / n
    return [x / rms for x in v]


def _start(shape, seed):
    """A velocity and the nonlinear term of an earlier one (complex128)."""
    g = _gen(seed)
    v, w = _velocity(shape, g), _velocity(shape, g)
    c0 = [_forward(x) for x in _crossed([torch.fft.ifftn(x) for x in w],
                                        [torch.fft.ifftn(x) for x in _curl(w)])]
    return v, c0


def _to(fields, dtype):
    return [f.to(dtype).contiguous() for f in fields]


def _ens_shapes(case):
    return [(32,) * 3] * case["n32"] + [(64,) * 3] * case["n64"] + [(128,) * 3] * case["n128"]


def _ens_nus(case):
    return [float(v) for v in np.geomspace(1 / 400, 1 / 100, len(_ens_shapes(case)))]


NU, DT = 1 / 200, 2.5e-4


def _fields(case, seed, count):
    g = _gen(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    return [torch.complex(torch.rand(shape, generator=g, device=DEV, dtype=torch.float64) * 2 - 1,
                          torch.rand(shape, generator=g, device=DEV, dtype=torch.float64) * 2 - 1)
            .to(_cdtype(case)) for _ in range(count)]


def _vectors(case, seed, count):
    """Fourier vectors of random real fields."""
    g = _gen(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    return [[_forward(torch.randn(shape, generator=g, device=DEV, dtype=torch.float64))
             .to(_cdtype(case)) for _ in range(3)] for _ in range(count)]


def _model_weights(seed):
    """He-style weights as the training starts from (numpy, float32 values)."""
    r = np.random.default_rng(seed)
    W1 = np.zeros((64, 16), np.float32)
    W1[:, :9] = r.standard_normal((64, 9)) * math.sqrt(2 / 9)
    W2 = (r.standard_normal((64, 64)) * math.sqrt(2 / 64)).astype(np.float32)
    w3 = (r.standard_normal(64) * math.sqrt(1 / 64)).astype(np.float32)
    b1, b2 = ((0.1 * r.standard_normal(64)).astype(np.float32) for _ in range(2))
    return W1, b1, W2, b2, w3, np.float32(0.1)


S_IN, S_OUT = 0.4, 1e-3


def _model(seed):
    return closure.MLPModel(*_model_weights(seed), s_in=S_IN, s_out=S_OUT, device=DEV)


def _les_csd2(case):
    return closure.smagorinsky_cs_delta2(0.17, case["n"] / 3)


def _samples(case, seed):
    """Model inputs, targets, weights of the strain, and a shuffled minibatch."""
    g = _gen(seed)
    m = case["rows"]
    A = torch.randn((m, 9), generator=g, device=DEV)
    X = torch.zeros((m, 16), device=DEV)
    X[:, :9] = A
    t = (0.3 * torch.randn(m, generator=g, device=DEV) + 0.5).clamp_min(0)
    w = A.square().mean(dim=1)
    idx = torch.randperm(m, generator=g, device=DEV)[:case["batch"]].to(torch.int32)
    return X.to(torch.bfloat16).contiguous(), t, w, idx.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "ns":
        shape = (case["nz"], case["ny"], case["nx"])
        v, c0 = _start(shape, seed)
        st["v"], st["c0"] = _to(v, _cdtype(case)), _to(c0, _cdtype(case))
        if case["bootstrap"]:
            st["w"] = _to(_curl(v), _cdtype(case))
            st["monitor"] = torch.zeros((case["steps"], 4), dtype=torch.float64).pin_memory()
        st["ns"] = S.NSStepper(shape, NU, DT, _cdtype(case), real=case["real"], tune=case["tune"])
    elif kind in ("fft", "poisson"):
        st["f"] = _fields(case, seed, case["fields"])
        if case["tune"]:
            S.fft3d_tune((case["nz"], case["ny"], case["nx"]), _cdtype(case), case["fields"])
    elif kind == "cross":
        st["a"], st["b"] = _vectors(case, seed, 2)
    elif kind == "project":
        st["v"], = _vectors(case, seed, 1)
    elif kind == "ens":
        shapes = _ens_shapes(case)
        st["ens"] = S.NSEnsemble(shapes, _ens_nus(case), DT, _cdtype(case), tune=case["tune"])
        st["state"] = [tuple(_to(x, _cdtype(case)) for x in _start(s, seed * 1000 + b))
                       for b, s in enumerate(shapes)]
    elif kind == "les":
        n = case["n"]
        v, c0 = _start((n,) * 3, seed)
        cut = _k2((n,) * 3) <= (n / 3) ** 2
        st["v"], st["c0"] = (_to([x * cut for x in f], _cdtype(case)) for f in (v, c0))
        st["ns"] = S.NSStepper((n,) * 3, NU, DT, _cdtype(case))
        st["model"] = _model(seed)
        st["ns"].set_closure(CLOSURES[case["model"]], cs_delta2=_les_csd2(case),
                             mlp=st["model"].packed, kc=n / 3)
    elif kind == "mlp":
        st["model"] = _model(seed)
        st["X"], st["t"], st["weight"], st["idx"] = _samples(case, seed)
    elif kind == "tracers":
        n, g = case["n"], _gen(seed)
        st["u"] = _to([torch.fft.ifftn(x) for x in _velocity((n,) * 3, g)], _cdtype(case))
        st["pos"] = torch.rand((case["particles"], 3), generator=g, device=DEV,
                               dtype=torch.float64) * (2 * math.pi)
    else:
        raise ValueError(kind)
    return st


# --------------------------------------------------------------------- one pass
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "ns" and case["bootstrap"]:
        ns = st["ns"]
        ns.bootstrap(st["v"], st["w"])
        for i in range(case["steps"]):
            ns.step(1)
            ns.stats_async(st["monitor"][i])
        return ns.state()
    if kind in ("ns", "les"):
        ns = st["ns"]
        ns.set_state(st["v"], st["c0"])
        ns.step(case["steps"])
        return ns.state()
    if kind == "fft":
        S.forward(st["f"], zero=False)
        S.inverse(st["f"])
        return st["f"]
    if kind == "poisson":
        S.forward(st["f"])
        for f in st["f"]:
            S.laplacian_inverse(f)
        S.inverse(st["f"])
        return st["f"]
    if kind == "cross":
        return S.cross(st["a"], st["b"])
    if kind == "project":
        v = st["v"]
        p = S.laplacian_inverse(S.divergence(v))
        grad = S.gradient(p)
        return {"v": [S.axpby(1.0, v[d], -1.0, grad[d]) for d in range(3)], "p": p}
    if kind == "ens":
        ens = st["ens"]
        for b, (v, c0) in enumerate(st["state"]):
            ens.set_state(b, v, c0)
        ens.step(case["steps"])
        got = [ens.state(b) for b in range(len(ens))]
        return {key: torch.cat([f.reshape(-1) for s in got for f in s[key]])
                for key in ("V1", "cross0")}
    if kind == "mlp":
        m = st["model"]
        return {"nut": m.infer(st["X"]),
                "grad": m.gradient(st["X"], st["t"], idx=st["idx"], weight=st["weight"])}
    if kind == "tracers":
        t = S.Tracers(st["pos"].clone())
        for _ in range(case["moves"]):
            t.move(st["u"], DT)
        return {"pos": t.pos, "vel": t.vel}
    raise ValueError(kind)


# --------------------------------------------------------------------- what a pass cannot avoid
def _esz(case):
    return 8 if case["dtype"] == "c64" else 16


def _fft_flops(n):
    return 5.0 * n * math.log2(n)


def _ns_work(n, esz, steps, real=False):
    """Per step: velocity and history read and written once, nine transforms and
    about a hundred operations of the update per mode."""
    part = 0.5 if real else 1.0
    return {"bytes": part * steps * 12.0 * n * esz,
            "flops": part * steps * (9 * _fft_flops(n) + 100.0 * n)}


def work(case):
    kind = case["kind"]
    if kind == "ns":
        return _ns_work(case["nx"] * case["ny"] * case["nz"], _esz(case), case["steps"],
                        case["real"])
    if kind in ("fft", "poisson"):
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 4.0 * n * _esz(case) * case["fields"],
                "flops": 2 * _fft_flops(n) * case["fields"]}
    if kind == "cross":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 9.0 * n * _esz(case), "flops": 9 * _fft_flops(n) + 24.0 * n}
    if kind == "project":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 7.0 * n * _esz(case), "flops": 40.0 * n}
    if kind == "ens":
        parts = [_ns_work(s[0] ** 3, _esz(case), case["steps"]) for s in _ens_shapes(case)]
        return {key: sum(p[key] for p in parts) for key in ("bytes", "flops")}
    if kind == "les":
        n = case["n"] ** 3
        w = _ns_work(n, _esz(case), case["steps"])
        per_point = 2 * (9 * 64 + 64 * 64 + 64) if case["model"] == "mlp" else 60
        w["flops"] += case["steps"] * (9 * _fft_flops(n) + per_point * n)
        return w
    if kind == "mlp":
        per_row = 2.0 * (9 * 64 + 64 * 64 + 64)
        return {"bytes": 36.0 * case["rows"] + 44.0 * case["batch"],
                "flops": per_row * (case["rows"] + 3.0 * case["batch"])}
    grid = min(case["n"] ** 3, 8 * case["particles"])
    return {"bytes": case["moves"] * (3.0 * _esz(case) * grid + 72.0 * case["particles"]),
            "flops": case["moves"] * 130.0 * case["particles"]}


# --------------------------------------------------------------------- in 64 bits
def _wide(fields):
    return [f.to(torch.complex128) for f in fields]


def _bf16(x):
    return torch.as_tensor(np.asarray(x, np.float32), device=DEV).to(torch.bfloat16).double()


def _network(weights, X):
    W1, b1, W2, b2, w3, b3 = weights
    h = torch.relu(X @ W1.T + b1)
    h = torch.relu(h @ W2.T + b2)
    return torch.nn.functional.softplus(h @ w3 + b3, threshold=700.0)


def _exact_weights(seed):
    """The packed model's values: BF16 weights, FP32 biases."""
    W1, b1, W2, b2, w3, b3 = _model_weights(seed)
    f = lambda x: torch.as_tensor(np.asarray(x, np.float64), device=DEV)  # noqa: E731
    return [_bf16(W1), f(b1), _bf16(W2), f(b2), _bf16(w3), f(b3)]


def _nonlinear(v, nu_t=None):
    """V x omega, with `nu_t` (a function of the real velocity gradient) the
    divergence of the eddy stress 2 nu_t S_ij added."""
    shape = v[0].shape
    u = [torch.fft.ifftn(x) for x in v]
    c = [_forward(x) for x in _crossed(u, [torch.fft.ifftn(x) for x in _curl(v)])]
    if nu_t is not None:
        A = [[torch.fft.ifftn(_ik(shape, j) * v[i]) for j in range(3)] for i in range(3)]
        nut = nu_t(A)
        for i in range(3):
            for j in range(3):
                c[i] += _ik(shape, j) * _forward(nut * (A[i][j] + A[j][i]))
    return c


def _advance(v, c0, nu, dt, steps, nu_t=None, cut=None):
    """AB2 / projection / Crank-Nicolson steps (exec/ns.cpp:167-217)."""
    shape = v[0].shape
    k, k2 = _k(shape), _k2(shape)
    inner = torch.where(k2 > 0, k2, torch.ones_like(k2))
    keep = None if cut is None else k2 <= cut * cut
    den = 1.0 + nu * dt / 2 * k2
    for _ in range(steps):
        c1 = _nonlinear(v, nu_t)
        if keep is not None:
            c1 = [c * keep for c in c1]
        F = [dt / 2 * (3 * c1[d] - c0[d]) for d in range(3)]
        lap = [-nu * dt / 2 * k2 * v[d] for d in range(3)]
        s = [v[d] + lap[d] + F[d] for d in range(3)]
        G = -1j * (k[0] * s[0] + k[1] * s[1] + k[2] * s[2]) / inner
        v = [(s[d] - 1j * k[d] * G) / den for d in range(3)]
        if keep is not None:
            v = [x * keep for x in v]
        c0 = c1
    return v, c0


def _bootstrapped(v, w, nu, dt):
    """The Forward-Euler first step (exec/ns.cpp:132-153)."""
    shape = v[0].shape
    k, k2 = _k(shape), _k2(shape)
    c = [_forward(x) for x in _crossed([torch.fft.ifftn(x) for x in v],
                                       [torch.fft.ifftn(x) for x in w])]
    t = [c[d] - nu * k2 * v[d] for d in range(3)]
    div = 1j * (k[0] * t[0] + k[1] * t[1] + k[2] * t[2])
    p = -div / torch.where(k2 > 0, k2, torch.ones_like(k2))
    return [v[d] + dt * (t[d] - 1j * k[d] * p) for d in range(3)], c


def exact(case, seed):
    st_kind = case["kind"]
    if st_kind == "ns":
        shape = (case["nz"], case["ny"], case["nx"])
        v, c0 = _start(shape, seed)
        if case["bootstrap"]:
            w = _wide(_to(_curl(v), _cdtype(case)))
            v, c0 = _bootstrapped(_wide(_to(v, _cdtype(case))), w, NU, DT)
        else:
            v, c0 = _wide(_to(v, _cdtype(case))), _wide(_to(c0, _cdtype(case)))
        v, c0 = _advance(v, c0, NU, DT, case["steps"])
        return {"V1": v, "omega1": _curl(v), "cross0": c0}
    if st_kind == "fft":
        return _wide(_fields(case, seed, case["fields"]))
    if st_kind == "poisson":
        k2 = _k2((case["nz"], case["ny"], case["nx"]))
        div = torch.where(k2 > 0, -k2, torch.ones_like(k2))
        return [torch.fft.ifftn(_forward(f) / div)
                for f in _wide(_fields(case, seed, case["fields"]))]
    if st_kind == "cross":
        a, b = ([torch.fft.ifftn(x) for x in _wide(v)] for v in _vectors(case, seed, 2))
        return [_forward(x) for x in _crossed(a, b)]
    if st_kind == "project":
        v = _wide(_vectors(case, seed, 1)[0])
        shape = v[0].shape
        k2 = _k2(shape)
        div = sum(_ik(shape, d) * v[d] for d in range(3))
        p = torch.where(k2 > 0, -div / torch.where(k2 > 0, k2, torch.ones_like(k2)), div)
        return {"v": [v[d] - _ik(shape, d) * p for d in range(3)], "p": p}
    if st_kind == "ens":
        V, C = [], []
        for b, (s, nu) in enumerate(zip(_ens_shapes(case), _ens_nus(case))):
            v, c0 = (_wide(_to(x, _cdtype(case))) for x in _start(s, seed * 1000 + b))
            v, c0 = _advance(v, c0, nu, DT, case["steps"])
            V += [f.reshape(-1) for f in v]
            C += [f.reshape(-1) for f in c0]
        return {"V1": torch.cat(V), "cross0": torch.cat(C)}
    if st_kind == "les":
        n = case["n"]
        cut = _k2((n,) * 3) <= (n / 3) ** 2
        v, c0 = (_wide(_to([x * cut for x in f], _cdtype(case))) for f in _start((n,) * 3, seed))
        if case["model"] == "mlp":
            weights = _exact_weights(seed)

            def nu_t(A):
                X = torch.zeros((n ** 3, 16), device=DEV, dtype=torch.float64)
                for q in range(9):
                    X[:, q] = S_IN * A[q // 3][q % 3].real.reshape(-1)
                return S_OUT * _network(weights, X).reshape((n,) * 3)
        else:
            def nu_t(A):
                s2 = sum((0.5 * (A[i][j].real + A[j][i].real)) ** 2
                         for i in range(3) for j in range(3))
                return _les_csd2(case) * torch.sqrt(2 * s2)
        v, c0 = _advance(v, c0, NU, DT, case["steps"], nu_t, n / 3)
        return {"V1": v, "omega1": _curl(v), "cross0": c0}
    if st_kind == "mlp":
        X, t, w, idx = _samples(case, seed)
        weights = [x.requires_grad_() for x in _exact_weights(seed)]
        loss = 0.0
        idx = idx.long()
        for part in idx.split(1 << 18):
            err = _network(weights, X[part].double()) - t[part].double()
            one = (w[part].double() * err.square()).sum() / idx.numel()
            one.backward()
            loss += float(one)
        grad = torch.cat([x.grad.reshape(-1) for x in weights] +
                         [torch.tensor([loss], device=DEV, dtype=torch.float64)])
        with torch.no_grad():
            nut = torch.cat([S_OUT * _network(weights, x.double()) for x in X.split(1 << 18)])
        return {"nut": nut, "grad": grad}
    n, g = case["n"], _gen(seed)
    u = [f.to(_cdtype(case)).real.double().reshape(-1)
         for f in (torch.fft.ifftn(x) for x in _velocity((n,) * 3, g))]
    x = torch.rand((case["particles"], 3), generator=g, device=DEV,
                   dtype=torch.float64) * (2 * math.pi)
    h = 2 * math.pi / n
    vel = torch.zeros_like(x)
    for _ in range(case["moves"]):
        i = (x / h).long().clamp(0, n - 2)
        r = (x - i * h) / h
        vel = torch.zeros_like(x)
        for dz in (0, 1):
            for dy in (0, 1):
                for dx in (0, 1):
                    at = (i[:, 0] + dx) + n * (i[:, 1] + dy) + n * n * (i[:, 2] + dz)
                    wt = ((r[:, 0] if dx else 1 - r[:, 0]) * (r[:, 1] if dy else 1 - r[:, 1]) *
                          (r[:, 2] if dz else 1 - r[:, 2]))
                    for d in range(3):
                        vel[:, d] += wt * u[d][at]
        x = x + vel * DT
        x = torch.where(x >= 2 * math.pi, x - 2 * math.pi,
                        torch.where(x <= 0, x + 2 * math.pi, x))
    return {"pos": x, "vel": vel}

"""What a user of this framework has it do, as cases that can be timed and checked.

`listed()` names the cases, `draw()` makes more of the same ranges, `prepare()` makes the
inputs and handles a user's program holds before the call, `run()` is one pass through the
public entry points, `work()` the bytes and operations a pass cannot do without, and
`exact()` what a pass returns, in 64 bits and plain torch.

Kinds of case:
  step      IMEXRK.TimeStep on one grid, one or several runs: a simulation that goes on from
            pass to pass
  linear    IMEXRK.TimeStepLinear about a frozen base: one Arnoldi or inverse-iteration action
  tangent   a tangent-linear batch (set_tangent): one block of Newton-Krylov Jacobian actions
  adjoint   IMEXRK.TimeStepAdjoint between two stored direct states
  ensemble  Ensemble.step over 2D runs on grids of different sizes
  krylov    one block Gram-Schmidt pass of the block Krylov solvers (Vecs.gram, Vecs.update)
  net       gradient of the continuation predictor over its training set (Net.gradient)
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

import stratiflow_b200 as sf

L1, L2, L3 = 2 * math.pi / 0.44, math.pi / 0.44, 10.0


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # the smallest call: one step of the small eigenvalue grid, where launches count
        dict(name="step2d_64", kind="step", N1=64, N2=1, N3=64, runs=1, steps=1, Re=1000.0, dt=0.01, bg="tanh"),
        # the plain 2D Kelvin-Helmholtz run, several steps a call
        dict(name="step2d_128", kind="step", N1=128, N2=1, N3=128, runs=1, steps=10, Re=1000.0, dt=0.01, bg="tanh"),
        # a parameter sweep in 2D, on a finer grid of ragged height
        dict(name="step2d_512_sweep", kind="step", N1=512, N2=1, N3=388, runs=6, steps=4, Re=1000.0, dt=0.01,
             bg="tanh"),
        # the block of Jacobian actions of the Newton-Krylov solver: 16 directions about one live base
        dict(name="tangent2d_256", kind="tangent", N1=256, N2=1, N3=256, runs=17, steps=4, Re=1000.0, dt=0.01,
             bg="tanh"),
        # the mixed ensemble: 64 runs over N1 in {64, 128, 256} and N3 in {128, 256, 384}
        dict(name="ensemble_64", kind="ensemble", pick=3, N1=256, N3=384, runs=64, steps=4, Re=1000.0, dt=0.01,
             bg="tanh"),
        # the reduced 3D grid of the tests
        dict(name="step3d_64", kind="step", N1=64, N2=32, N3=64, runs=1, steps=4, Re=4000.0, dt=0.005, bg="holmboe"),
        # an ordinary 3D run, two at once, on a ragged height
        dict(name="step3d_128", kind="step", N1=128, N2=64, N3=180, runs=2, steps=2, Re=4000.0, dt=0.005,
             bg="holmboe"),
        # the benchmark's 3D shear layer
        dict(name="step3d_256", kind="step", N1=256, N2=128, N3=384, runs=1, steps=1, Re=4000.0, dt=0.005,
             bg="holmboe"),
        # a linearised evolution about a frozen 3D state
        dict(name="linear3d_128", kind="linear", N1=128, N2=64, N3=192, runs=2, steps=2, Re=4000.0, dt=0.005,
             bg="holmboe"),
        # one adjoint step of the 3D mixing optimisation
        dict(name="adjoint3d_128", kind="adjoint", N1=128, N2=64, N3=128, runs=1, steps=1, Re=4000.0, dt=0.005,
             bg="holmboe"),
        # one Gram-Schmidt pass of a block of 16 against a basis of 320 vectors
        dict(name="krylov2d_256", kind="krylov", N1=256, N2=1, N3=256, basis=320, block=16, Re=1000.0, dt=0.01,
             bg="tanh"),
        # the predictor's training set of 13 triples: loss and gradient, forward and backward
        dict(name="predictor_13", kind="net", c0=1024, c1=256, c2=256, c3=256, c4=512, Z=256, batch=13),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pow2(rng, lo, hi):
    return 2 ** rng.randint(int(math.log2(lo)), int(math.log2(hi)))


MOST_POINTS = 256 * 128 * 384   # grid points x runs x steps of the largest listed step


def draw(rng: random.Random):
    kind = rng.choice(["step", "step", "step", "linear", "tangent", "adjoint", "ensemble", "krylov", "net"])
    if kind == "net":
        c = [16 * rng.randint(8, 64), 32 * rng.randint(3, 8), 32 * rng.randint(3, 8), 32 * rng.randint(3, 8),
             16 * rng.randint(6, 32)]
        return dict(kind="net", c0=c[0], c1=c[1], c2=c[2], c3=c[3], c4=c[4], Z=4 * rng.randint(16, 64),
                    batch=rng.randint(2, 13))
    dim3 = kind in ("step", "linear", "adjoint") and rng.random() < 0.55
    Re, dt, bg = (4000.0, 0.005, "holmboe") if dim3 else (1000.0, 0.01, "tanh")
    if kind == "ensemble":
        return dict(kind="ensemble", pick=rng.randint(10, 10 ** 6), N1=_pow2(rng, 64, 256), N3=4 * _log(rng, 24, 96),
                    runs=_log(rng, 4, 64), steps=rng.randint(1, 4), Re=Re, dt=dt, bg=bg)
    if kind == "krylov":
        return dict(kind="krylov", N1=_pow2(rng, 64, 256), N2=1, N3=4 * _log(rng, 16, 64), basis=_log(rng, 16, 320),
                    block=rng.randint(1, 16), Re=Re, dt=dt, bg=bg)
    while True:
        if dim3:
            N1, N2 = _pow2(rng, 32, 256), _pow2(rng, 16, 128)
        else:
            N1, N2 = _pow2(rng, 32, 512), 1
        N3 = 4 * _log(rng, 9, 96)
        runs = _log(rng, 1, 3) if dim3 else _log(rng, 1, 32)
        if kind == "tangent":
            runs = max(2, runs)
        steps = 1 if kind == "adjoint" else rng.randint(1, 4)
        share = 4 if kind in ("linear", "adjoint", "tangent") else 1
        if share * N1 * N2 * N3 * runs * steps <= MOST_POINTS and N2 <= 2 * N1:
            return dict(kind=kind, N1=N1, N2=N2, N3=N3, runs=runs, steps=steps, Re=Re, dt=dt, bg=bg)


def _members(case):
    """(N1, N3) of the ensemble's runs: the case's largest grid and its halves and parts of a third."""
    rng = random.Random(case["pick"])
    n1 = [max(32, case["N1"] // d) for d in (1, 2, 4)]
    n3 = [max(36, case["N3"] * p // 12 * 4) for p in (1, 2, 3)]
    return [(rng.choice(n1), rng.choice(n3)) for _ in range(case["runs"])]


# ----------------------------------------------------------------- inputs --
def _grid(N):
    """z (Dirichlet levels), zf (Neumann levels), DY, DYF of the stretched grid."""
    z, zf = sf.vertical_points(L3, N), sf.vertical_points_fractional(L3, N)
    dy, dyf = np.zeros(N), np.zeros(N)
    dy[1:] = zf[1:] - zf[:-1]
    dyf[1:N - 1] = z[2:] - z[1:N - 1]
    dyf[N - 1], dyf[0] = dyf[N - 2], dyf[1]
    return z, zf, dy, dyf


def _modes(N1, N2):
    """kx [K1] and ky [K2] of the kept modes, K1, K2 and the number of non-negative ky."""
    K1, Ky = N1 // 3, (N2 // 3 if N2 > 1 else 1)
    K2 = 2 * Ky - 1 if N2 > 1 else 1
    j2 = np.array([q if q < Ky else q - K2 for q in range(K2)], dtype=float)
    return np.arange(K1) * 2 * math.pi / L1, j2 * 2 * math.pi / L2, K1, K2, Ky


def _states(N1, N2, N3, runs, seed, amp=0.05):
    """Seeded states of a run in progress, in the kept layout [runs][5][N3][plane] on the GPU:
    smooth in z, confined to the shear layer, a spectrum that falls off with the wavenumber over
    all kept modes, real fields (Hermitian at kx = 0) and a velocity without divergence on the
    staggered grid (u1 = dA/dz, u2 = dB/dz, u3 = -(dA/dx + dB/dy))."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dev, M = "cuda", 6
    z, zf, _, dyf = (torch.tensor(a, device=dev) for a in _grid(N3))
    kx, ky, K1, K2, Ky = _modes(N1, N2)
    kx, ky = torch.tensor(kx, device=dev), torch.tensor(ky, device=dev)
    c = torch.randn((runs, 4, M, K2, K1), generator=gen, device=dev, dtype=torch.complex64).to(torch.complex128)
    # kx = 0: conjugate pairs in ky, a real mean
    if K2 > 1:
        c[..., Ky:, 0] = c[..., 1:Ky, 0].flip(-1).conj()
    c[..., 0, 0] = c[..., 0, 0].real.to(torch.complex128)
    j = torch.arange(K1, device=dev, dtype=torch.float64)[None, :] ** 2
    j2 = (ky * L2 / (2 * math.pi))[:, None] ** 2
    c = c * (amp / (1 + (j + j2) / 16) ** 2)
    m = torch.arange(M, device=dev, dtype=torch.float64)

    def basis(x):
        return torch.cos(m[:, None] * x[None, :] * 0.8 + m[:, None]) * torch.exp(-x * x / 4) / (1 + m[:, None])

    bz, bf = basis(z), basis(zf)
    bz[:, :3] = 0
    bz[:, -2:] = 0
    bf[:, 0] = 0
    bf[:, -1] = 0
    plane = (K1 * K2 + 15) // 16 * 16
    out = torch.zeros((runs, 5, N3, plane), device=dev, dtype=torch.complex64)

    def put(f, x):
        out[:, f, :, :K1 * K2] = x.reshape(runs, N3, K1 * K2).to(torch.complex64)

    def up(x):   # Dirichlet -> Neumann difference
        d = torch.zeros_like(x)
        d[:, 1:-1] = (x[:, 2:] - x[:, 1:-1]) / dyf[1:-1, None, None]
        return d

    a = torch.einsum("rmqk,mz->rzqk", c[:, 0], bz.to(c.dtype))
    put(0, up(a))
    u3 = -1j * kx * a
    if N2 > 1:
        b = torch.einsum("rmqk,mz->rzqk", c[:, 1], bz.to(c.dtype))
        put(1, up(b))
        u3 = u3 - 1j * ky[:, None] * b
    put(2, u3)
    put(3, torch.einsum("rmqk,mz->rzqk", c[:, 2], bf.to(c.dtype)))
    put(4, torch.einsum("rmqk,mz->rzqk", c[:, 3], bf.to(c.dtype)))
    return out


def _ri(case):
    n = case.get("runs", 1)
    return [0.16 if n == 1 else 0.05 + 0.2 * r / (n - 1) for r in range(n)]


def _solver(case, N1, N2, N3, runs):
    s = sf.IMEXRK(N1, N2, N3, L1, L2, L3, case["Re"], 1.0, case["dt"], nrun=runs)
    U, dB = sf.background_profile(case["bg"], L3, N3)
    ri = _ri(case) if case["kind"] == "step" else [0.12] * runs
    for r in range(runs):
        s.set_ri(r, ri[r])
        s.SetBackground(r, U, dB)
    return s


class _Device:
    """A device buffer of the framework, which its owner frees: the tensor made of it keeps the owner."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<c8", data=(ptr, False), version=3)


def _view(ptr, shape, owner):
    return torch.as_tensor(_Device(ptr, shape, owner), device="cuda")


def _current(s, owner=None):
    """The flow, as SaveFlow writes it: u1, u2, u3, b of every run. Not p, the sum of the projections'
    q / h: the rounding of the divergence over h makes its fifth digit, in any order of evaluation;
    its gradient is in the velocity."""
    return _view(s.state_device_ptr()[0], s.kept_shape, owner or s)[:, :4]


def _net_params(case, seed):
    rng = np.random.default_rng(seed)
    parts, ch = [], [case["c%d" % i] for i in range(5)]
    for ci, co in zip(ch[:-1], ch[1:]):
        parts += [rng.standard_normal(co * 5 * ci, dtype=np.float32) * np.float32(math.sqrt(2 / (5 * ci))),
                  rng.standard_normal(co, dtype=np.float32) * np.float32(0.05)]
    x = rng.standard_normal((case["batch"], case["Z"], ch[0]), dtype=np.float32)
    t = rng.standard_normal((case["batch"], case["Z"], ch[-1]), dtype=np.float32)
    return ch, np.concatenate(parts), x, t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "net":
        ch, w, x, t = _net_params(case, seed)
        net = sf.Net(ch, case["Z"], case["batch"])
        net.set_params(w)
        net.set_data(x, t)
        return dict(case=case, net=net)
    if kind == "ensemble":
        grids = _members(case)
        e = sf.Ensemble(grids, (L1, L3, case["Re"], 1.0), case["dt"])
        for r, (m, (n1, n3)) in enumerate(zip(e.members, grids)):
            U, dB = sf.background_profile(case["bg"], L3, n3)
            m.set_ri(0, _ri(case)[r])
            m.SetBackground(0, U, dB)
            x = _states(n1, 1, n3, 1, seed * 1000 + r)
            torch.cuda.synchronize()
            m.set_state_device(x.data_ptr())
            m.synchronize()
        return dict(case=case, ensemble=e)
    N1, N2, N3 = case["N1"], case["N2"], case["N3"]
    if kind == "krylov":
        na, nb = case["basis"], case["block"]
        s = _solver(case, N1, N2, N3, nb)
        v = sf.Vecs(s, na + nb)
        for i in range(0, na + nb, nb):   # the basis, then the block: nb states at a time
            i = min(i, na)
            x = _states(N1, N2, N3, nb, seed * 1000 + i)
            torch.cuda.synchronize()
            s.set_state_device(x.data_ptr())
            s.synchronize()
            if i < na:
                v.from_run(i, 0, min(nb, na - i))
        x = _states(N1, N2, N3, nb, seed * 1000 + na)
        torch.cuda.synchronize()
        s.set_state_device(x.data_ptr())
        s.synchronize()
        v.synchronize()
        return dict(case=case, solver=s, vecs=v)
    runs = case["runs"]
    s = _solver(case, N1, N2, N3, runs)
    x = _states(N1, N2, N3, runs, seed * 1000)
    st = dict(case=case, solver=s, x=x)
    if kind == "linear":
        st["base"] = _states(N1, N2, N3, runs, seed * 1000 + 1, amp=0.1)
        torch.cuda.synchronize()
        for r in range(runs):
            if sf.load_library().sf_set_base_device(s.handle, r, ctypes.c_void_p(st["base"][r].data_ptr())):
                raise sf.SFError("sf_set_base_device")
    if kind == "adjoint":
        st["below"], st["above"] = sf.Vecs(s, runs), sf.Vecs(s, runs)
        for k, v in enumerate((st["below"], st["above"])):
            d = _states(N1, N2, N3, runs, seed * 1000 + 2 + k, amp=0.1)
            torch.cuda.synchronize()
            s.set_state_device(d.data_ptr())
            s.synchronize()
            v.from_run(0, 0, runs)
            v.synchronize()
    if kind == "tangent":
        s.set_tangent(1)
    torch.cuda.synchronize()
    s.set_state_device(x.data_ptr())
    s.synchronize()
    return st


# ----------------------------------------------------------------- a pass --
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "net":
        g, loss = st["net"].gradient()
        return dict(gradient=g, loss=loss)
    if kind == "ensemble":
        e = st["ensemble"]
        e.step(case["steps"])
        e.synchronize()
        return [_current(m, e) for m in e.members]
    s = st["solver"]
    if kind == "krylov":
        v, na, nb = st["vecs"], case["basis"], case["block"]
        v.from_run(na, 0, nb)
        c = v.gram(0, na, v, na, nb, 0.12)
        v.update(na, nb, -1.0, v, 0, na, c)
        v.synchronize()
        p = ctypes.c_void_p()
        if sf.load_library().sf_vecs_device(v._h, na, ctypes.byref(p)):
            raise sf.SFError("sf_vecs_device")
        return dict(gram=c, block=_view(p.value, (nb,) + v.shape, v))
    if kind == "step":
        s.TimeStep(case["steps"])
    else:   # an operator applied to given states
        s.set_state_device(st["x"].data_ptr())
        if kind == "linear":
            s.TimeStepLinear(case["steps"])
        elif kind == "tangent":
            s.TimeStep(case["steps"])
        else:
            s.TimeStepAdjoint(st["below"], st["above"])
    s.synchronize()
    return _current(s)


def _step_work(N1, N2, N3, runs, steps, extra_in=0, products=None):
    K1, K2 = _modes(N1, N2)[2:4]
    nf = 5 if N2 > 1 else 4
    S = N3 * K1 * K2 * 8 * runs
    n = N1 * N2
    ffts = (nf - 1) + (products or (11 if N2 > 1 else 6))
    flops = 3 * steps * runs * N3 * (ffts * 2.5 * n * math.log2(n) + 40 * n + 40 * nf * K1 * K2)
    return {"bytes": (2 * nf + extra_in) * S, "flops": flops}


def work(case):
    """Each input state read once and each result written once; the transforms' and solves' operations."""
    kind = case["kind"]
    if kind == "net":
        ch = [case["c%d" % i] for i in range(5)]
        rows = case["batch"] * case["Z"]
        w = [5 * a * b for a, b in zip(ch[:-1], ch[1:])]
        return {"bytes": 8 * (sum(w) + sum(ch[1:])) + 4 * rows * (ch[0] + ch[-1]),
                "flops": 2.0 * rows * (3 * sum(w) - w[0])}
    if kind == "ensemble":
        ws = [_step_work(n1, 1, n3, 1, case["steps"]) for n1, n3 in _members(case)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    N1, N2, N3 = case["N1"], case["N2"], case["N3"]
    if kind == "krylov":
        K1, K2 = _modes(N1, N2)[2:4]
        na, nb, S = case["basis"], case["block"], N3 * K1 * K2 * 8
        nf = 4 if N2 > 1 else 3
        return {"bytes": S * (nf * (na + nb) + (nf + 1) * nb), "flops": 8.0 * nf * N3 * K1 * K2 * na * nb}
    if kind == "linear":
        return _step_work(N1, N2, N3, case["runs"], case["steps"], extra_in=4 if N2 > 1 else 3)
    if kind == "adjoint":
        d = N2 > 1
        return _step_work(N1, N2, N3, case["runs"], 1, extra_in=8 if d else 6, products=32 if d else 17)
    return _step_work(N1, N2, N3, case["runs"], case["steps"])


# -------------------------------------------------------- 64-bit results --
class _Flow64:
    """The scheme in 64-bit torch: fields [runs][N3][K2][K1], three stages of explicit terms,
    Crank-Nicolson diffusion and projection."""

    def __init__(self, case, N1, N2, N3, ri):
        dev = "cuda"
        t = lambda a: torch.tensor(np.asarray(a, dtype=np.float64), device=dev)  # noqa: E731
        self.N1, self.N2, self.N3 = N1, N2, N3
        kx, ky, self.K1, self.K2, self.Ky = _modes(N1, N2)
        self.P = self.K1 * self.K2
        self.kx, self.ky = 1j * t(kx), 1j * t(ky)[:, None]
        self.k2 = -(t(kx)[None, :] ** 2 + t(ky)[:, None] ** 2)
        _, _, dy, dyf = _grid(N3)
        self.dy, self.dyf = dy, dyf
        self.Re, self.dt = case["Re"], case["dt"]
        self.h = [self.dt * 8 / 15, self.dt * 2 / 15, self.dt * 5 / 15]
        self.ri = t(ri).reshape(-1, 1, 1, 1)
        U, dB = sf.background_profile(case["bg"], L3, N3)
        self.U, self.dB = t(U).reshape(-1, 1, 1), t(dB).reshape(-1, 1, 1)
        j = np.arange(N3)
        self.D2N, self.D2D = np.zeros((3, N3)), np.zeros((3, N3))
        i = j[1:N3 - 1]
        self.D2N[0, i], self.D2N[2, i] = 1 / dy[i] / dyf[i], 1 / dy[i + 1] / dyf[i]
        self.D2N[1] = -self.D2N[0] - self.D2N[2]
        i = j[2:N3 - 1]
        self.D2D[0, i], self.D2D[2, i] = 1 / dyf[i - 1] / dy[i], 1 / dyf[i] / dy[i]
        self.D2D[1] = -self.D2D[0] - self.D2D[2]
        col = lambda a: t(a).reshape(-1, 1, 1)  # noqa: E731
        self.band = {k: [col(r) for r in b] for k, b in (("N", self.D2N), ("D", self.D2D))}
        one = np.ones(N3)
        w = lambda lo, di: (col(lo[1:]), col(di[1:]))  # noqa: E731
        d1 = np.where(j >= 1, dy, 1.0)
        low = np.concatenate([[1.0], dyf[:-1]])
        self.w = {"full": w(dyf / (2 * d1), low / (2 * d1)), "tilde": w(low / (2 * d1), dyf / (2 * d1)),
                  "bar": w(0.5 * one, 0.5 * one)}
        inv = np.where(j >= 2, 1 / d1, 0.0)
        self.wdn = w(-inv, inv)
        self.wdd = col(np.where(j >= 1, 1 / dyf, 0.0))
        self.fac = {("lap",): self._factor(self.D2N, 1.0, 0.0, "lap")}
        for k in range(3):
            for bc, band in (("N", self.D2N), ("D", self.D2D)):
                self.fac[(bc, k)] = self._factor(band, -0.5 * self.h[k] / self.Re, 1.0, bc)

    def _factor(self, band, scale, one, bc):
        """Thomas factors of one + scale (d2z + k2) with the end rows of its boundary condition."""
        N = self.N3
        a, c = scale * band[0].copy(), scale * band[2].copy()
        b = one + scale * (torch.tensor(band[1], device="cuda").reshape(-1, 1, 1) + self.k2)
        rows = (0, 1, 2, N - 2, N - 1) if bc == "D" else (0, 1, N - 2, N - 1)
        for r in rows:
            a[r], c[r], b[r] = 0, 0, 1
        if bc != "D":
            c[1], a[N - 2], b[N - 2] = -1, 1, -1
        a = torch.tensor(a, device="cuda").reshape(-1, 1, 1).expand_as(b).clone()
        c = torch.tensor(c, device="cuda").reshape(-1, 1, 1).expand_as(b).clone()
        if bc == "lap":   # the mean: q fixed at the lower end
            c[1, 0, 0] = 0
        C, D = torch.zeros_like(b), torch.zeros_like(b)
        D[0] = 1 / b[0]
        C[0] = c[0] * D[0]
        for j in range(1, N):
            D[j] = 1 / (b[j] - a[j] * C[j - 1])
            C[j] = c[j] * D[j]
        return [x.unsqueeze(-1) for x in (-a * D, D, -C)]

    def solve(self, key, d, bc):
        aD, D, C = self.fac[key]
        N = self.N3
        d[:, 0], d[:, 1], d[:, N - 2], d[:, N - 1] = 0, 0, 0, 0
        if bc == "D":
            d[:, 2] = 0
        x = torch.view_as_real(d).transpose(0, 1).contiguous() * D.unsqueeze(1)
        for j in range(1, N):
            x[j].addcmul_(aD[j], x[j - 1])
        for j in range(N - 2, -1, -1):
            x[j].addcmul_(C[j], x[j + 1])
        return torch.view_as_complex(x.transpose(0, 1).contiguous())

    def nodal(self, f):
        s = f.shape[0]
        g = torch.zeros((s, self.N3, self.N2, self.N1 // 2 + 1), dtype=torch.complex128, device=f.device)
        g[:, :, :self.Ky, :self.K1] = f[:, :, :self.Ky]
        if self.K2 > 1:
            g[:, :, self.N2 - self.Ky + 1:, :self.K1] = f[:, :, self.Ky:]
        return torch.fft.irfft2(g, s=(self.N2, self.N1), norm="forward")

    def modal(self, x):
        g = torch.fft.rfft2(x, norm="forward")[..., :self.K1]
        return g if self.K2 == 1 else torch.cat([g[:, :, :self.Ky], g[:, :, self.N2 - self.Ky + 1:]], 2)

    # vertical operators on axis 1
    def R(self, kind, f):
        g = torch.zeros_like(f)
        lo, di = self.w[kind]
        g[:, 1:] = lo * f[:, :-1] + di * f[:, 1:]
        return g

    def Rdir(self, f):
        g = 0.5 * f
        g[:, :-1] += 0.5 * f[:, 1:]
        return g

    def dn(self, f):   # Neumann -> Dirichlet
        g = torch.zeros_like(f)
        g[:, 1:] = self.wdn[0] * f[:, :-1] + self.wdn[1] * f[:, 1:]
        return g

    def dd(self, f):   # Dirichlet -> Neumann
        g = -f
        g[:, :-1] += f[:, 1:]
        return g * self.wdd

    def d2(self, bc, f):
        lo, di, up = self.band[bc]
        g = di * f
        g[:, 1:] += (lo[1:] * f[:, :-1])
        g[:, :-1] += (up[:-1] * f[:, 1:])
        return g

    def buoyancy(self, s):
        b = s["b"].clone()
        b[:, :, 0, 0] = 0
        return dict(u1=0, u2=0, u3=self.ri * self.R("full", b), b=-self.dB * self.Rdir(s["u3"]))

    def rhs(self, s, base=None):
        """Explicit terms; with base (modal), linearised about it."""
        r, m, R = self.buoyancy(s), self.modal, self.R
        names = ("u1", "u2", "u3", "b") if self.N2 > 1 else ("u1", "u3", "b")
        n = {k: self.nodal(s[k]) for k in names}
        if base is None:
            n["u1"] = n["u1"] + self.U
            pr = lambda f, g: f(n[g[0]]) * (n[g[1]] if g[2] is None else g[2](n[g[1]]))  # noqa: E731
        else:
            q = {k: self.nodal(base[k]) for k in names}
            q["u1"] = q["u1"] + self.U

            def pr(f, g):
                e = g[2] or (lambda x: x)
                return f(n[g[0]]) * e(q[g[1]]) + f(q[g[0]]) * e(n[g[1]])
        idf = lambda x: x  # noqa: E731
        bar, til = (lambda x: R("bar", x)), (lambda x: R("tilde", x))
        kx, ky = self.kx, self.ky
        r["u1"] = r["u1"] - kx * m(pr(idf, ("u1", "u1", None))) - m(self.dd(pr(bar, ("u1", "u3", None))))
        r["u3"] = r["u3"] - kx * m(pr(til, ("u1", "u3", None))) - self.dn(m(pr(self.Rdir, ("u3", "u3", self.Rdir))))
        r["b"] = r["b"] - m(self.dd(pr(bar, ("b", "u3", None)))) - kx * m(pr(idf, ("u1", "b", None)))
        if self.N2 > 1:
            x = m(pr(idf, ("u1", "u2", None)))
            r["u1"] = r["u1"] - ky * x
            r["u2"] = (r["u2"] - ky * m(pr(idf, ("u2", "u2", None))) - m(self.dd(pr(bar, ("u2", "u3", None))))
                       - kx * x)
            r["u3"] = r["u3"] - ky * m(pr(til, ("u2", "u3", None)))
            r["b"] = r["b"] - ky * m(pr(idf, ("u2", "b", None)))
        return r

    def rhs_adjoint(self, s, d):
        """Explicit terms of the adjoint about the direct state d (modal, U included in u1)."""
        m, t, R, kx, ky = self.modal, self.nodal, self.R, self.kx, self.ky
        three = self.N2 > 1
        names = ("u1", "u2", "u3", "b") if three else ("u1", "u3", "b")
        n, T = {k: t(s[k]) for k in names}, {k: t(d[k]) for k in names}
        mean = lambda f: f[:, :, 0, 0].real[:, :, None, None]  # noqa: E731
        full = lambda x: R("full", x)  # noqa: E731
        bF = 0.5 * (T["u3"] - mean(d["u3"])) + self.ri * self.Rdir(n["u3"])
        f3 = 0.5 * (T["b"] - mean(d["b"]))
        r1 = kx * m(n["u1"] * T["u1"]) + m(self.dd(R("bar", n["u1"]) * T["u3"]))
        r3 = kx * m(R("tilde", T["u1"]) * n["u3"]) + self.dn(m(self.Rdir(n["u3"]) * self.Rdir(T["u3"])))
        rB = m(self.dd(R("bar", n["b"]) * T["u3"])) + kx * m(n["b"] * T["u1"])
        f1 = -t(kx * d["u1"]) * n["u1"] - self.Rdir(t(kx * d["u3"]) * n["u3"]) - t(kx * d["b"]) * n["b"]
        f3 = f3 - t(self.dn(d["u1"])) * full(n["u1"]) - full(t(self.dd(d["u3"]))) * n["u3"]
        f3 = f3 - t(self.dn(d["b"])) * full(n["b"])
        r = {}
        if three:
            r2 = (ky * m(n["u2"] * T["u2"]) + m(self.dd(R("bar", n["u2"]) * T["u3"])) + kx * m(n["u2"] * T["u1"]))
            r3 = r3 + ky * m(R("tilde", T["u2"]) * n["u3"])
            r1 = r1 + ky * m(n["u1"] * T["u2"])
            rB = rB + ky * m(n["b"] * T["u2"])
            f1 = f1 - t(kx * d["u2"]) * n["u2"]
            f2 = (-t(ky * d["u1"]) * n["u1"] - t(ky * d["u2"]) * n["u2"] - self.Rdir(t(ky * d["u3"]) * n["u3"])
                  - t(ky * d["b"]) * n["b"])
            f3 = f3 - t(self.dn(d["u2"])) * full(n["u2"])
            r["u2"] = r2 + m(f2)
        r.update(u1=r1 + m(f1), u3=r3 + m(f3), b=rB + m(bF))
        return r

    def stage(self, k, s, r, old):
        h, z, bt = self.h[k], (0.0, -17 / 8, -5 / 4)[k], (1.0, 25 / 8, 9 / 4)[k]
        grad = dict(u1=self.kx * s["p"], u2=self.ky * s["p"], u3=self.dn(s["p"]), b=0)
        c, out = 0.5 * h / self.Re, {}
        for f in ("u1", "u2", "u3", "b"):
            if f == "u2" and self.N2 == 1:
                out[f] = s[f]
                continue
            bc = "D" if f == "u3" else "N"
            x = s[f] - h * grad[f] + h * bt * r[f] + c * (self.k2 * s[f] + self.d2(bc, s[f]))
            if old is not None:
                x = x + h * z * old[f]
            out[f] = self.solve((bc, k), x, bc)
        div = self.kx * out["u1"] + self.dd(out["u3"])
        if self.N2 > 1:
            div = div + self.ky * out["u2"]
        q = self.solve(("lap",), div, "N")
        out["u1"] = out["u1"] - self.kx * q
        if self.N2 > 1:
            out["u2"] = out["u2"] - self.ky * q
        out["u3"] = out["u3"] - self.dn(q)
        out["p"] = s["p"] + q / h
        return out

    def unpack(self, x):
        x = x[..., :self.P].to(torch.complex128).reshape(x.shape[0], 5, self.N3, self.K2, self.K1)
        return {k: x[:, i] for i, k in enumerate(("u1", "u2", "u3", "b", "p"))}

    def pack(self, s, plane):
        x = torch.stack([s[k] for k in ("u1", "u2", "u3", "b")], 1)
        out = torch.zeros(x.shape[:3] + (plane,), dtype=x.dtype, device=x.device)
        out[..., :self.P] = x.reshape(x.shape[:3] + (self.P,))
        return out


def _part(s, lo, hi):
    return {k: v[lo:hi] for k, v in s.items()}


def _evolve64(case, N1, N2, N3, x, ri, base=None, ends=None, tangent=False):
    """u1, u2, u3, b of the states x after the case's steps, kept layout, complex128."""
    f = _Flow64(case, N1, N2, N3, ri)
    s = f.unpack(x)
    q = None if base is None else f.unpack(base)
    for _ in range(case["steps"]):
        old, frac = None, 0.0
        for k in range(3):
            if ends is not None:
                lo, hi = (f.unpack(e) for e in ends)
                d = {n: (1 - frac) * hi[n] + frac * lo[n] for n in ("u1", "u2", "u3", "b")}
                d["u1"][:, :, 0, 0] += f.U.reshape(1, -1)
                r = f.rhs_adjoint(s, d)
                frac += f.h[k] / f.dt
            elif tangent:
                # run 0 is the live base of the other runs
                R = next(iter(s.values())).shape[0]
                ri_all = f.ri
                f.ri = ri_all[:1]
                b0 = _part(s, 0, 1)
                r0 = f.rhs(b0)
                f.ri = ri_all[1:]
                r1 = f.rhs(_part(s, 1, R), {n: v.expand(R - 1, -1, -1, -1) for n, v in b0.items()})
                f.ri = ri_all
                zero = torch.zeros_like(s["u2"])
                r = {n: torch.cat([r0[n], r1[n]]) if torch.is_tensor(r0[n]) else zero for n in r0}
            else:
                r = f.rhs(s, q)
            s = f.stage(k, s, r, old)
            old = r
    return f.pack(s, x.shape[-1])


def _net64(case, seed):
    ch, w, x, t = _net_params(case, seed)
    dev = "cuda"
    w = torch.tensor(w, device=dev, dtype=torch.float64).requires_grad_()
    a, o = torch.tensor(x, device=dev, dtype=torch.float64), 0
    B, Z = a.shape[:2]
    for l, (ci, co) in enumerate(zip(ch[:-1], ch[1:])):
        W = w[o:o + co * 5 * ci].reshape(co, 5 * ci)
        o += co * 5 * ci
        bias = w[o:o + co]
        o += co
        p = torch.nn.functional.pad(a, (0, 0, 2, 2))
        a = torch.cat([p[:, k:k + Z] for k in range(5)], -1).reshape(B * Z, 5 * ci) @ W.T + bias
        a = a.reshape(B, Z, co)
        if l < 3:
            a = torch.relu(a)
    loss = (a - torch.tensor(t, device=dev, dtype=torch.float64)).square().mean()
    loss.backward()
    return dict(gradient=w.grad, loss=float(loss))


def exact(case, seed):
    kind = case["kind"]
    if kind == "net":
        return _net64(case, seed)
    if kind == "ensemble":
        grids, ri = _members(case), _ri(case)
        out = [None] * len(grids)
        for n1, n3 in sorted(set(grids)):   # the runs of one grid together
            who = [r for r, g in enumerate(grids) if g == (n1, n3)]
            x = torch.cat([_states(n1, 1, n3, 1, seed * 1000 + r) for r in who])
            y = _evolve64(case, n1, 1, n3, x, [ri[r] for r in who])
            for i, r in enumerate(who):
                out[r] = y[i:i + 1]
        return out
    N1, N2, N3 = case["N1"], case["N2"], case["N3"]
    if kind == "krylov":
        na, nb = case["basis"], case["block"]
        rows = [_states(N1, N2, N3, nb, seed * 1000 + i)[:min(nb, na - i)] for i in range(0, na, nb)]
        V = torch.cat(rows).to(torch.complex128)
        W = _states(N1, N2, N3, nb, seed * 1000 + na).to(torch.complex128)
        z, zf, _, _ = _grid(N3)
        wn, wd = np.zeros(N3), np.zeros(N3)
        wn[1:N3 - 1] = z[2:] - z[1:N3 - 1]
        wd[2:N3 - 1] = zf[2:N3 - 1] - zf[1:N3 - 2]
        # the quadrature weights as the framework holds them, in 32 bits
        wt = torch.tensor(np.stack([wn, wn, wd, wn]).astype(np.float32), device="cuda", dtype=torch.float64)
        wt = wt * torch.tensor([1.0, 1.0, 1.0, 0.12], device="cuda", dtype=torch.float64)[:, None]
        wm = torch.full((V.shape[-1],), 2.0, device="cuda", dtype=torch.float64)
        wm[0] = 1.0
        w = wt[None, :, :, None] * wm
        c = torch.view_as_real(V[:, :4] * w).reshape(na, -1) @ torch.view_as_real(W[:, :4]).reshape(nb, -1).T
        out = W.clone()
        out[:, :4] -= torch.einsum("ik,ifzm->kfzm", c.to(V.dtype), V[:, :4])
        return dict(gram=c, block=out)
    runs = case["runs"]
    x = _states(N1, N2, N3, runs, seed * 1000)
    base = ends = None
    if kind == "linear":
        base = _states(N1, N2, N3, runs, seed * 1000 + 1, amp=0.1)
    if kind == "adjoint":
        ends = [_states(N1, N2, N3, runs, seed * 1000 + 2 + k, amp=0.1) for k in range(2)]
    ri = _ri(case) if kind == "step" else [0.12] * runs
    return _evolve64(case, N1, N2, N3, x, ri, base, ends, kind == "tangent")

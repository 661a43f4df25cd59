"""The work a user of this framework has it do, as cases that can be timed.

Every case goes through the public Python mirror (Solver, Ensemble, Krylov).
`listed()` names the standing cases, `draw()` gives others of the same ranges,
`prepare()` builds what a user's program holds before the call, `run()` is one
pass, `work()` what a pass cannot do without, and `exact()` the same results
in plain torch (complex128, cuFFT line transforms) without this package's code.

Kinds of case:
  rk3       RK3_SSP steps of one grid (optionally FP32 mode, tuned tiles, or
            with the main loop's diagnostics read back after the step)
  ensemble  RK3_SSP steps of a batch of instances, each with its own dt and Re
  jvp       RK3_SSP_UV tangent steps (one product of the exponential map)
  matvec    one linearised product J(u) v on packed Krylov vectors
  fft       FFTN_Device and iFFTN_Device of one field
  arnoldi   one Arnoldi factorisation over the 1-D Laplacian
Fields are the seeded Kolmogorov recipe of the benchmarks: the laminar profile
(Re/16) sin 4y plus a divergence-free |k|^-2 perturbation, forced by sin 4y,
dt from CFL 0.3 of the laminar peak (0.003 in the FP32 mode, whose state and
update are FP64: a step's FP32 rounding scales with dt, and at this dt it
stays below what FP64 outputs are compared to).
"""
import math

import numpy as np
import torch

from ns3dperiodic_b200 import Ensemble, Krylov, Solver

PI = 3.141592653589793238462643383279502884197169399375105820974944592307816406
EXTENTS = (16, 24, 32, 48, 64, 96, 128, 192, 256, 384)


def _case(name, kind, nx=0, ny=0, nz=0, **kw):
    c = {"name": name, "kind": kind}
    if nx:
        c.update(nx=nx, ny=ny or nx, nz=nz or nx)
    c.update(kw)
    return c


def listed():
    return [
        # the exact-solution test's grid: the smallest call, one step at a time,
        # as a program that looks at the state after every step makes it
        _case("rk3_32", "rk3", 32, re=20.0, steps=1),
        # the reference's main loop: a step, then energy / dissipation / divergence on the host
        _case("loop_64", "rk3", 64, re=50.0, steps=1, diagnostics=True),
        # the Kolmogorov run's grid, ten steps between two looks at the state
        _case("rk3_128", "rk3", 128, re=100.0, steps=10),
        # the headline benchmark: 256^3 FP64, tiles tuned as bench.py tunes them
        _case("rk3_256", "rk3", 256, re=400.0, steps=1, tune=True),
        # the largest grid of the precision study
        _case("rk3_512", "rk3", 512, re=400.0, steps=1),
        # the FP32 mode of the precision study
        _case("rk3_256_fp32", "rk3", 256, re=400.0, steps=1, fp32=True),
        # a box with a different, partly non-power-of-two extent per direction
        _case("rk3_384x48x192", "rk3", 384, 48, 192, re=50.0, steps=2),
        # one product of the exponential map of the restarted Arnoldi run: 20 tangent steps
        _case("jvp_64", "jvp", 64, re=50.0, steps=20),
        # one linearised product of Newton-Krylov / Arnoldi on packed vectors
        _case("matvec_96", "matvec", 96, re=100.0),
        # one grid's batch of the mixed-N ensemble, FP32 mode, tuned
        _case("ensemble_96x12_fp32", "ensemble", 96, batch=12, steps=2, fp32=True, tune=True),
        # plain transforms there and back, as a program that looks at physical fields makes them
        _case("fft_256", "fft", 256),
        # the Krylov self-test: Gram-Schmidt over 2.3 million unknowns, 30 columns
        _case("arnoldi_2300000x30", "arnoldi", n=2300000, m=30),
    ]


def draw(rng):
    """One more case: grids from 16 to 384 points per direction, to 256^3 in all."""
    kind = rng.choice(["rk3", "rk3", "rk3", "ensemble", "jvp", "matvec", "fft", "arnoldi"])
    if kind == "arnoldi":
        return {"kind": kind, "n": int(math.exp(rng.uniform(math.log(2e4), math.log(2.3e6)))) | 1,
                "m": rng.randint(8, 30)}
    top = {"ensemble": 96, "jvp": 128, "matvec": 192}.get(kind, 256)
    want = math.exp(rng.uniform(math.log(16.0), math.log(float(top))))
    if kind == "ensemble" or rng.random() < 0.4:
        n = min(EXTENTS, key=lambda e: abs(math.log(e / want)))
        dims = (n, n, n)
    else:
        while True:
            dims = tuple(rng.choice([e for e in EXTENTS if want / 4 <= e <= want * 4])
                         for _ in range(3))
            if dims[0] * dims[1] * dims[2] <= top ** 3:
                break
    c = {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2]}
    if kind == "fft":
        return c
    c["re"] = round(rng.uniform(0.6, 1.0) * min(dims), 3)
    if kind == "ensemble":
        del c["re"]
        c["batch"] = rng.randint(2, max(2, min(24, int(8 * (96.0 / dims[0]) ** 2))))
        c["steps"] = rng.randint(1, 4)
        c["fp32"] = rng.random() < 0.5
    elif kind == "rk3":
        c["steps"] = rng.randint(1, 8)
        c["fp32"] = rng.random() < 0.3
        c["diagnostics"] = rng.random() < 0.3
    elif kind == "jvp":
        c["steps"] = rng.randint(1, 10)
    return c


# ---------------------------------------------------------------------------
# seeded inputs, on the GPU
# ---------------------------------------------------------------------------
def _dims(case):
    return int(case["nx"]), int(case["ny"]), int(case["nz"])


def _signed(n):
    j = torch.arange(n, device="cuda", dtype=torch.float64)
    return torch.where(j >= n // 2, j - n, j)


def _waves(dims):
    nx, ny, nz = dims
    return (_signed(nx)[:, None, None], _signed(ny)[None, :, None],
            torch.arange(nz // 2 + 1, device="cuda", dtype=torch.float64)[None, None, :])


def _perturbation(dims, gen):
    """Unit-norm divergence-free pure-imaginary spectrum, |k|^-2 on 1 <= |k| <= 8."""
    nx, ny, nz = dims
    k = _waves(dims)
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    amp = torch.where((k2 >= 1.0) & (k2 <= 64.0), 1.0 / k2.clamp(min=1.0), torch.zeros_like(k2))
    amp[nx // 2] = 0.0
    amp[:, ny // 2] = 0.0
    w = []
    for _ in range(3):
        a = torch.randn(k2.shape, generator=gen, device="cuda", dtype=torch.float64).mul_(amp)
        for l in (0, nz // 2):  # odd planes: a real field's spectrum
            p = a[:, :, l].clone()
            a[:, :, l] = 0.5 * (p - torch.roll(torch.flip(p, (0, 1)), (1, 1), (0, 1)))
        w.append(a)
    del amp
    kw = (k[0] * w[0] + k[1] * w[1] + k[2] * w[2]) / k2.clamp(min=1.0)
    for c in range(3):
        w[c].addcmul_(k[c].expand_as(kw), kw, value=-1.0)
    norm = math.sqrt(sum(float(a.square().sum()) for a in w))
    return [torch.complex(torch.zeros_like(a), a.div_(norm)) for a in w]


def _forcing(dims):
    nx, ny, nz = dims
    F = [torch.zeros((nx, ny, nz // 2 + 1), dtype=torch.complex128, device="cuda")
         for _ in range(3)]
    F[0][0, 4, 0] = -0.5j * nx * ny * nz
    F[0][0, ny - 4, 0] = 0.5j * nx * ny * nz
    return F


def _flow(dims, re, gen):
    """Laminar profile plus a perturbation of a tenth of its norm."""
    nx, ny, nz = dims
    U = _perturbation(dims, gen)
    a = 0.5 * nx * ny * nz * re / 16.0
    for u in U:
        u.mul_(0.1 * a * math.sqrt(2.0))
    U[0][0, 4, 0] += -1j * a
    U[0][0, ny - 4, 0] += 1j * a
    return U


def _dt(case, re):
    cfl = 0.003 if case.get("fp32") else 0.3
    return cfl * (2.0 * PI / max(_dims(case))) / (re / 16.0)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _ensemble_params(case, seed):
    r = np.random.default_rng(int(seed))
    re = r.uniform(0.5, 1.0, int(case["batch"])) * float(case["nx"])
    return [_dt(case, float(x)) for x in re], [float(x) for x in re]


def _inputs(case, seed):
    """The tensors of a case, before any handle of the framework exists."""
    kind, gen = case["kind"], _gen(seed)
    if kind == "arnoldi":
        return {"f": torch.randn(int(case["n"]), generator=gen, device="cuda",
                                 dtype=torch.float64)}
    dims = _dims(case)
    if kind == "fft":
        x = torch.randn(dims, generator=gen, device="cuda", dtype=torch.float64)
        return {"x": x, "X": _perturbation(dims, gen)[0]}
    if kind == "ensemble":
        dt, re = _ensemble_params(case, seed)
        each = [_flow(dims, r, gen) for r in re]
        return {"U": [torch.stack([e[c] for e in each]) for c in range(3)],
                "F": _forcing(dims), "dt": dt, "re": re}
    s = {"U": _flow(dims, float(case["re"]), gen), "F": _forcing(dims),
         "dt": _dt(case, float(case["re"])), "re": float(case["re"])}
    if kind == "jvp":
        s["V"] = _perturbation(dims, gen)
    elif kind == "matvec":
        v = torch.cat([p.imag.reshape(-1)[1:] for p in _perturbation(dims, gen)])
        s["v"] = v.contiguous()
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    s["case"] = case
    if kind == "arnoldi":
        n, m = int(case["n"]), int(case["m"])
        s["kr"] = Krylov(n, m)
        s["A"] = s["kr"].laplace_map()
        s["V"] = torch.zeros((m, n), dtype=torch.float64, device="cuda")
        s["r"] = torch.empty_like(s["f"])
        s["H"] = np.zeros((m, m))
        return s
    dims = _dims(case)
    if kind == "ensemble":
        h = Ensemble(int(case["batch"]), *dims)
        if case.get("fp32"):
            h.set_precision("fp32")
        h.set_params(s["dt"], s["re"])
    else:
        h = Solver(*dims)
        if case.get("fp32"):
            h.precision = "fp32"
    if kind != "fft":
        h.set_forcing(s["F"])
    if case.get("tune"):
        h.autotune()
    s["h"] = h
    if kind == "fft":
        s["Y"] = torch.empty_like(s["X"])
        s["y"] = torch.empty_like(s["x"])
    elif kind == "matvec":
        s["w"] = torch.empty_like(s["v"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "rk3":
        s["h"].rk3_ssp(s["U"], s["dt"], s["re"], int(case["steps"]))
        if case.get("diagnostics"):
            return s["U"], s["h"].diagnostics(s["U"])
        return s["U"]
    if kind == "ensemble":
        return s["h"].rk3_steps(s["U"], int(case["steps"]))
    if kind == "jvp":
        return s["h"].rk3_ssp_uv(s["U"], s["V"], s["dt"], s["re"], int(case["steps"]))
    if kind == "matvec":
        return s["h"].matvec_reduced(s["U"], s["v"], s["re"], out=s["w"])
    if kind == "fft":
        return s["h"].fftn(s["x"], out=s["Y"]), s["h"].ifftn(s["X"], out=s["y"])
    s["r"].copy_(s["f"])  # a new start vector: the driver consumes it
    s["kr"].arnoldi(s["A"], s["V"], s["H"], s["r"], 0, int(case["m"]))
    return s["V"], s["H"], s["r"]


def work(case):
    """State read and written once per step (fields, Krylov columns) and the
    arithmetic of the real transforms the formulation needs (2.5 N log2 N each)."""
    if case["kind"] == "arnoldi":
        n, m = case["n"], case["m"]
        # the basis and the residual written once; two Gram-Schmidt sweeps per column
        return {"bytes": 8.0 * n * (m + 2), "flops": 8.0 * n * m * (m + 1) / 2.0}
    nx, ny, nz = _dims(case)
    field = 16.0 * nx * ny * (nz // 2 + 1)
    points = float(nx * ny * nz)
    fft = 2.5 * points * math.log2(points)
    steps = int(case.get("steps", 1)) * int(case.get("batch", 1))
    if case["kind"] == "fft":
        return {"bytes": 2.0 * (field + 8.0 * points), "flops": 2.0 * fft}
    if case["kind"] == "matvec":
        return {"bytes": 3.0 * field + 2.0 * 1.5 * field, "flops": 27.0 * fft}
    if case["kind"] == "jvp":
        return {"bytes": 12.0 * field * steps, "flops": (2 * 27.0 + 3 * 15.0) * fft * steps}
    return {"bytes": 6.0 * field * steps, "flops": 45.0 * fft * steps}


# ---------------------------------------------------------------------------
# the same results in plain torch
# ---------------------------------------------------------------------------
class _Plain:
    """The reference's discretisation on one grid of the 2 pi box."""

    def __init__(self, dims):
        self.dims = dims
        nx, ny, nz = dims
        mz = nz // 2 + 1
        self.k = _waves(dims)
        # the kept modes, by the reference's own sequence of operations
        m = np.where(np.arange(nx) >= nx // 2, np.arange(nx) - nx, np.arange(nx))
        n = np.where(np.arange(ny) >= ny // 2, np.arange(ny) - ny, np.arange(ny))
        length = 2.0 * PI
        kx, ky, kz = (a * 2 * PI / length for a in (m, n, np.arange(mz)))
        tx = kx * kx / ((2 * nx * PI / length) * (2 * nx * PI / length))
        ty = ky * ky / ((2 * ny * PI / length) * (2 * ny * PI / length))
        tz = kz * kz / ((2 * mz * PI / length) * (2 * mz * PI / length))
        keep = np.sqrt((tx[:, None, None] + ty[None, :, None]) + tz[None, None, :]) < 2.0 / 3.0
        keep[0, 0, 0] = False
        self.mask = torch.from_numpy(keep).to("cuda")

    def k2(self):
        return self.k[0] ** 2 + self.k[1] ** 2 + self.k[2] ** 2

    def inverse(self, X):
        w = torch.fft.ifft(torch.fft.ifft(X, dim=0), dim=1)
        w[:, :, 0].imag.zero_()
        w[:, :, -1].imag.zero_()
        return torch.fft.irfft(w, n=self.dims[2], dim=2)

    def forward(self, x):
        return torch.fft.fft(torch.fft.fft(torch.fft.rfft(x, dim=2), dim=1), dim=0)

    def physical(self, U):
        return [self.inverse(u * self.mask) for u in U]

    def gradient(self, u, axis):
        return self.inverse((1j * self.k[axis]) * (u * self.mask))

    def spectrum(self, q):
        Q = self.forward(q)
        Q.real.zero_()
        Q[0, 0, 0] = 0
        return Q

    def advection(self, U):
        u = self.physical(U)
        return [self.spectrum(sum(u[j] * self.gradient(U[i], j) for j in range(3)))
                for i in range(3)]

    def tangent(self, U, V):
        u, v = self.physical(U), self.physical(V)
        return [self.spectrum(sum(v[j] * self.gradient(U[i], j) + u[j] * self.gradient(V[i], j)
                                  for j in range(3))) for i in range(3)]

    def project(self, Q):
        """AM.Q - Q, the negated divergence-free part."""
        kq = (self.k[0] * Q[0] + self.k[1] * Q[1] + self.k[2] * Q[2]) / self.k2().clamp(min=1.0)
        return [self.k[i] * kq - Q[i] for i in range(3)]

    def euler(self, U, Q, F, dt, re):
        P = self.project(Q)
        G = 1.0 - self.k2() * dt / re
        return [dt * P[i] + G * U[i] + (dt * F[i] if F else 0.0) for i in range(3)]

    def rk3(self, U, F, dt, re):
        a = self.euler(U, self.advection(U), F, dt, re)
        b = self.euler(a, self.advection(a), F, dt, re)
        a = [0.75 * U[i] + 0.25 * b[i] for i in range(3)]
        b = self.euler(a, self.advection(a), F, dt, re)
        return [U[i] / 3.0 + 2.0 / 3.0 * b[i] for i in range(3)]

    def rk3_uv(self, U, V, F, dt, re):
        w = self.euler(V, self.tangent(U, V), None, dt, re)
        U = self.rk3(U, F, dt, re)
        w = self.euler(w, self.tangent(U, w), None, dt, re)
        return U, [0.5 * V[i] + 0.5 * w[i] for i in range(3)]

    def linearised(self, U, V, re):
        P = self.project(self.tangent(U, V))
        return [P[i] - self.k2() / re * V[i] for i in range(3)]


def _exact_arnoldi(f, m):
    n = f.numel()
    V = torch.zeros((m, n), dtype=torch.float64, device="cuda")
    H = np.zeros((m, m))
    for j in range(m):
        beta = float(torch.linalg.vector_norm(f))
        V[j] = f / beta
        if j:
            H[j, j - 1] = beta
        f = torch.roll(V[j], -1) - 2.0 * V[j] + torch.roll(V[j], 1)
        f[0] = 0.0
        for _ in range(2):
            c = V[:j + 1] @ f
            f = f - V[:j + 1].T @ c
            H[:j + 1, j] += c.cpu().numpy()
    return V, H, f


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "arnoldi":
        return _exact_arnoldi(s["f"], int(case["m"]))
    p = _Plain(_dims(case))
    if kind == "fft":
        return p.forward(s["x"]), p.inverse(s["X"])
    if kind == "matvec":
        nc = p.mask.numel()
        V = []
        for c in range(3):
            a = torch.zeros(nc, dtype=torch.float64, device="cuda")
            a[1:] = s["v"][c * (nc - 1):(c + 1) * (nc - 1)]
            V.append(torch.complex(torch.zeros_like(a), a).reshape(p.mask.shape))
        return torch.cat([w.imag.reshape(-1)[1:] for w in p.linearised(s["U"], V, s["re"])])
    if kind == "ensemble":
        out = [[], [], []]
        for b in range(int(case["batch"])):
            U = [u[b] for u in s["U"]]
            for _ in range(int(case["steps"])):
                U = p.rk3(U, s["F"], s["dt"][b], s["re"][b])
            for c in range(3):
                out[c].append(U[c])
        return [torch.stack(o) for o in out]
    U = s["U"]
    if kind == "jvp":
        V = s["V"]
        for _ in range(int(case["steps"])):
            U, V = p.rk3_uv(U, V, s["F"], s["dt"], s["re"])
        return U, V
    for _ in range(int(case["steps"])):
        U = p.rk3(U, s["F"], s["dt"], s["re"])
    return (U, (None, None, None)) if case.get("diagnostics") else U

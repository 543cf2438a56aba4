"""Workloads of the pipe-flow timestep library, for timing it and checking it.

`listed()` gives the standing cases, `draw(rng)` one more of the same ranges,
`prepare` what a program holds before the call, `run` one pass through the
public entry points, `work` the bytes and operations a pass cannot do without
and `exact` the pass's outputs in plain 64-bit torch, from the equations.

Kinds of pass:

  steps      a lone pipe: state vector in, main-loop timesteps (corrector to
             convergence), state vector out; optionally with a util plug-in
  adaptive   a fresh variable-dt run on the pipe's memory: matrices, then
             timesteps whose dt (and matrices) follow the CFL and corrector limits
  map        the time-T map of the Newton-Krylov search (one GMRES product):
             new dt and matrices, ndts one-corrector steps, the shift back
  batch      many uneven pipes advanced together
  serve      requests from host states through the continuous-batching server
  coll2phys  the velocity on the physical grid through the transform that
             works on the caller's own device memory

A state vector holds 8 header doubles, then per mode and radial point
(ur, ut, uz) Re/Im, scaled as newton.f90:567-602 does with scaleU = 1.
"""
import ctypes as C
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "softx-d-17-00015_b200"))
import pipeflow as P  # noqa: E402
from pipeflow.newton import Orbit  # noqa: E402

KL = 4
DECAY = 10.0  # of the seeded spectra, from the mean mode to the last one: that of a resolved run
PHYS = ("N", "K", "M", "Mp", "Re", "alpha", "dt")
# Carreau-Yasuda: rho, radius, mu_0, mu_inf, lambda, n, a; Coriolis: Ek0, phi
PLUGINS = {"carreau_yasuda": (P._lib.PF_UTIL_CARREAU_YASUDA, (1000.0, 0.01, 0.05, 0.0035, 3.3, 0.36, 2.0)),
           "coriolis": (P._lib.PF_UTIL_CORIOLIS, (0.5, 0.7))}


def _pipe(N, K, M, Mp=1, Re=2000.0, alpha=1.25, dt=0.01, mixed=False):
    return dict(N=N, K=K, M=M, Mp=Mp, Re=Re, alpha=alpha, dt=dt, mixed=mixed)


def listed():
    return [
        # the smallest run (the smoke test's size): launches and latency only
        dict(_pipe(16, 4, 4), name="steps-small", kind="steps", plugin="", steps=4, energy=1e-3),
        # the reference's CPU-runnable case, the plain FP64 drop-in
        dict(_pipe(40, 24, 16), name="steps-cfg1", kind="steps", plugin="", steps=4, energy=1e-3),
        # one pipe of the batched mix alone, in mixed precision
        dict(_pipe(48, 64, 24, Re=2400.0, alpha=1.1, mixed=True), name="steps-mixed", kind="steps", plugin="",
             steps=2, energy=1e-3),
        # the large FP64 drop-in: transforms of 384 x 144, two-fold symmetric
        dict(_pipe(64, 128, 48, Mp=2, Re=5300.0, alpha=0.5, dt=0.005), name="steps-cfg2", kind="steps", plugin="",
             steps=2, energy=1e-2),
        # sizes picked without a look at the transform lengths: 3K = 60, 3M = 33, odd N
        dict(_pipe(37, 20, 11, Re=2500.0, alpha=1.1), name="steps-odd", kind="steps", plugin="", steps=2,
             energy=1e-3),
        # the shear-thinning plug-in inside the step
        dict(_pipe(40, 24, 16), name="steps-carreau", kind="steps", plugin="carreau_yasuda", steps=2, energy=1e-3),
        # a variable-dt run: dt grows at once and is cut back, with new matrices each time
        dict(_pipe(40, 24, 16), name="adaptive-cfg1", kind="adaptive", plugin="", steps=4, energy=1e-3),
        # one product of the Newton-Krylov search at the drop-in's size
        dict(_pipe(40, 24, 16), name="map-cfg1", kind="map", plugin="", steps=16, energy=1e-3),
        # the benchmark's ensemble: 64 uneven pipes in mixed precision
        dict(name="batch64-mixed", kind="batch", pipes=64, mix=3, small=False, mixed=True, steps=2, energy=1e-3),
        # a small FP64 ensemble, sizes of the tests
        dict(name="batch8-fp64", kind="batch", pipes=8, mix=5, small=True, mixed=False, steps=4, energy=1e-3),
        # ten time-T requests of uneven length, the last four arriving while the first run
        dict(name="serve10", kind="serve", pipes=10, mix=7, small=True, mixed=True, steps=4, energy=1e-4),
        # a velocity field on the grid of the mix's largest shape
        dict(_pipe(64, 64, 32), name="coll2phys", kind="coll2phys", fields=3),
    ]


NOALLOC_SCRATCH = 24 * 1024 * 1024  # PF_NOALLOC_SCRATCH_BYTES of the C ABI
BUILT = (4, 5, 6, 8, 12, 16, 24, 32, 48, 64, 96, 128)  # 3K, 3M with built kernels


def _smooth(n):
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def _draw_pipe(rng, most_modes):
    """Sizes spread over their logarithm; half the transform lengths as a user who looked them up would pick them."""
    while True:
        def length(hi):
            n = int(round(math.exp(rng.uniform(math.log(4), math.log(hi)))))
            if rng.random() < 0.5:
                n = min(BUILT, key=lambda b: abs(b - n))
            return n
        N, K, M = rng.randint(14, 64), length(96), length(48)
        if _smooth(K) and _smooth(M) and N * K * M <= most_modes:
            return _pipe(N, K, M, Mp=rng.choice((1, 1, 2)), Re=round(rng.uniform(1800, 3000), 1),
                         alpha=round(rng.uniform(0.8, 1.6), 3), dt=rng.choice((0.01, 0.01, 0.005)))


def draw(rng):
    kind = rng.choice(("steps", "steps", "steps", "steps", "adaptive", "map", "batch", "batch", "serve", "coll2phys"))
    if kind == "steps":
        d = dict(_draw_pipe(rng, 60000), kind=kind, mixed=rng.random() < 0.4, steps=rng.randint(1, 3),
                 plugin=rng.choice(("", "", "", "", "", "carreau_yasuda", "coriolis")), energy=1e-3)
        if d["plugin"] == "coriolis":  # that plug-in has no azimuthal symmetry
            d["Mp"] = 1
        return d
    if kind == "adaptive":
        return dict(_draw_pipe(rng, 20000), kind=kind, plugin="", mixed=rng.random() < 0.3, steps=rng.randint(2, 5),
                    energy=1e-3)
    if kind == "map":
        return dict(_draw_pipe(rng, 20000), kind=kind, plugin="", mixed=rng.random() < 0.3,
                    steps=rng.randint(4, 24), energy=1e-3)
    if kind == "coll2phys":
        while True:
            N, K, M = rng.randint(10, 64), rng.choice(BUILT), rng.choice(BUILT)
            if N * K * M * 48 + 65536 <= NOALLOC_SCRATCH:
                return dict(_pipe(N, K, M), kind=kind, fields=rng.choice((1, 3)))
    n = rng.randint(2, 8)
    return dict(kind=kind, pipes=n, mix=rng.randrange(1 << 20), small=rng.random() < 0.5, mixed=rng.random() < 0.7,
                steps=rng.randint(2, 4), energy=1e-4 if kind == "serve" else 1e-3)


def _mix(case):
    """The pipes of a batch or a request stream."""
    rng = np.random.default_rng(case["mix"])
    ns, ks, ms = ((20, 24, 32, 48), (6, 8, 16, 32), (5, 8, 12, 24)) if case["small"] else \
        ((32, 48, 64), (16, 32, 64), (12, 24, 32))
    out = []
    for i in range(case["pipes"]):
        d = _pipe(int(rng.choice(ns)), int(rng.choice(ks)), int(rng.choice(ms)))
        d["Re"], d["alpha"] = float(rng.uniform(1800, 3000)), float(rng.uniform(0.8, 1.6))
        # a request stream brings FP64 Krylov evaluations among mixed-precision runs
        d["mixed"] = bool(case["mixed"]) and not (case["kind"] == "serve" and i % 3 == 2)
        out.append(d)
    return out


def _nsteps(case, i):
    """Steps of pipe i: requests differ in length, the pipes of a batch do not."""
    return case["steps"] - i % 3 if case["kind"] == "serve" and case["steps"] > 3 else case["steps"]


def _cfg(d, **more):
    return P.PipeConfig(**{k: d[k] for k in PHYS}, precision=P.PF_PREC_MIXED if d["mixed"] else P.PF_PREC_FP64, **more)


# ------------------------------------------------- the equations, in plain torch
DEV = "cuda"


def _weights(deriv, x, x0):
    """Finite-difference weights of the deriv-th derivative at x0 from the points x."""
    lo, hi = min(x0, x.min()), max(x0, x.max())
    A = np.polynomial.chebyshev.chebvander(2 * (x - lo) / (hi - lo) - 1, len(x) - 1)
    at = 2 * (x0 - lo) / (hi - lo) - 1
    d = np.array([np.polynomial.chebyshev.chebval(at, np.polynomial.chebyshev.chebder(e, deriv))
                  for e in np.eye(len(x))])
    return np.linalg.solve(A.T, d) * (2.0 / (hi - lo)) ** deriv


_GRIDS = {}


def _grid(N):
    """Radial points, d/dr, the radial Laplacian, the axis and wall rows and the r dr weights (numpy)."""
    if N not in _GRIDS:
        n2 = N + int(math.sqrt(N))
        r = np.array([0.5 * (1 + math.cos(math.pi * (n2 - n) / n2)) for n in range(n2 - N + 1, n2 + 1)])
        for _ in range(10):
            s = 1.5 * r[0] - 0.5 * r[1]
            r = r * (1 + s) - s
        D1, D2, w = np.zeros((N, N)), np.zeros((N, N)), np.zeros(N)
        for n in range(N):
            lo, hi = max(0, n - KL), min(N, n + KL + 1)
            D1[n, lo:hi], D2[n, lo:hi] = _weights(1, r[lo:hi], r[n]), _weights(2, r[lo:hi], r[n])
            up = r[min(n + 1, N - 1)] - r[n]
            dn = (r[n - 1] if n else 0.0) - r[n]
            c = e = 1.0
            for i in range(1, hi - lo + 1):
                c, e = c * up / i, e * dn / i
                w[lo:hi] += 0.5 * (c - e) * _weights(i - 1, r[lo:hi], r[n]) * r[n]
        axis = [_weights(i, r[:KL + 1], 0.0) for i in (0, 1)]
        wall = [_weights(i, r[-KL - 1:], 1.0) for i in (0, 1)]
        _GRIDS[N] = r, D1, D2 + D1 / r[:, None], axis, wall, w
    return _GRIDS[N]


class _Flow:
    """Fields are complex128 (N, H) tensors, modes in the order m, then k from -(K-1) (from 0 for m = 0)."""

    def __init__(self, d):
        self.d, self.N, self.K, self.M, self.dt = d, d["N"], d["K"], d["M"], d["dt"]
        r, D1, lap, self.axis, self.wall, w = _grid(self.N)
        t = lambda a: torch.tensor(np.asarray(a), dtype=torch.float64, device=DEV)  # noqa: E731
        self.r_np, self.r, self.D1, self.lap, self.w = r, t(r)[:, None], t(D1).to(torch.complex128), t(lap), t(w)
        self.wallz = t(self.wall[1])
        m, k = [], []
        for i in range(self.M):
            for j in range(0 if i == 0 else 1 - self.K, self.K):
                m.append(i)
                k.append(j)
        self.mi, self.ki = torch.tensor(m, device=DEV), torch.tensor(k, device=DEV)
        self.m, self.k = t(m) * d["Mp"], t(k) * d["alpha"]
        self.U, self.Up = 1 - self.r ** 2, -2 * self.r
        self.implicit, self.dterr = 0.51, 1e-5
        self.LN = None

    # --- state vectors
    def scale(self):
        s = torch.sqrt(self.w.abs())[:, None] * (4 / (4 + self.k.abs() + self.m))[None]
        z = s.clone()
        z[:, 0] = torch.sqrt(self.w.abs())
        return torch.stack([s, s, z], -1)  # (N, H, 3)

    def pack(self, u):
        v = torch.view_as_real(torch.stack(list(u), -1) * self.scale()).permute(1, 0, 2, 3)
        return torch.cat([torch.zeros(8, dtype=torch.float64, device=DEV), v.reshape(-1)])

    def seeded(self, seed, energy):
        """curl of a random vector potential of a resolved run's spectrum, scaled to energy times the laminar one."""
        g = np.random.default_rng(seed).standard_normal((3, 2, self.mi.numel()))
        amp = torch.exp(-DECAY * (self.ki.abs() / self.K + self.mi / self.M))
        am = self.m[None]
        rt = self.r ** (am + 1) * (1 - self.r ** 2) ** 2
        A = [torch.tensor(g[c, 0] + 1j * g[c, 1], device=DEV) * amp * (rt if c < 2 else rt * self.r) for c in range(3)]
        u = self.sym(self.curl(A))
        e = sum(float((self.w @ (x.abs() ** 2)).sum() - 0.5 * (self.w @ (x[:, 0].abs() ** 2))) for x in u)
        e *= 4 * math.pi ** 2 / self.d["alpha"]
        s = math.sqrt(energy * math.pi ** 2 / (3 * self.d["alpha"]) / e)
        return [x * s for x in u]

    # --- spectral operators
    def curl(self, u):
        ur, ut, uz = u
        mr = self.m / self.r
        return [1j * (mr * uz - self.k * ut), 1j * self.k * ur - self.D1 @ uz,
                ut / self.r + self.D1 @ ut - 1j * mr * ur]

    def grad(self, p):
        return [self.D1 @ p, 1j * self.m / self.r * p, 1j * self.k * p]

    def sym(self, u):
        u = [x.clone() for x in u]
        u[0][:, 0] = 0
        u[1][:, 0] = u[1][:, 0].real + 0j
        u[2][:, 0] = u[2][:, 0].real + 0j
        return u

    def phys(self, c):
        """(N, Th, Z) on the 3/2 grid."""
        N, K, M, Z = self.N, self.K, self.M, 3 * self.K
        X = torch.zeros(N, M, Z, dtype=torch.complex128, device=DEV)
        X[:, 0, :K] = c[:, :K]
        if K > 1:
            X[:, 0, 2 * K + 1:] = c[:, 1:K].flip(1).conj()
        rest = c[:, K:].reshape(N, M - 1, 2 * K - 1)
        X[:, 1:, :K] = rest[:, :, K - 1:]
        X[:, 1:, 2 * K + 1:] = rest[:, :, :K - 1]
        Y = torch.fft.ifft(X, dim=2, norm="forward").transpose(1, 2)
        F = torch.zeros(N, Z, 3 * M // 2 + 1, dtype=torch.complex128, device=DEV)
        F[:, :, :M] = Y
        F[:, :, 0] = F[:, :, 0].real + 0j
        return torch.fft.irfft(F, n=3 * M, dim=2, norm="forward").transpose(1, 2)

    def spec(self, p):
        N, K, M = self.N, self.K, self.M
        X = torch.fft.fft(torch.fft.rfft(p.transpose(1, 2), dim=2)[:, :, :M].transpose(1, 2), dim=2)
        X = X / (9 * K * M)
        rest = torch.cat([X[:, 1:, 2 * K + 1:], X[:, 1:, :K]], 2)
        return torch.cat([X[:, 0, :K], rest.reshape(N, -1)], 1)

    # --- the step
    def nonlinear(self, u, plugin=""):
        v = [self.phys(x) for x in u]
        q = [self.phys(x) for x in self.curl(u)]
        N = [self.spec(v[1] * q[2] - v[2] * q[1]), self.spec(v[2] * q[0] - v[0] * q[2]),
             self.spec(v[0] * q[1] - v[1] * q[0])]
        N = [x - 1j * self.k * self.U * y for x, y in zip(N, u)]
        N[2] = N[2] - self.Up * u[0]
        pr0 = (self.wallz @ u[2][-KL - 1:, 0].real) / -2
        N[2][:, 0] += 4 * pr0 / self.d["Re"]
        self.v = v
        if plugin:
            N = [x + y for x, y in zip(N, getattr(self, plugin)(u, v))]
        return N

    def coriolis(self, u, v):
        ek, phi = PLUGINS["coriolis"][1]
        th = 2 * math.pi / (3 * self.M) * torch.arange(3 * self.M, dtype=torch.float64, device=DEV)[:, None]
        o = [math.sin(phi) * torch.cos(th), -math.sin(phi) * torch.sin(th), math.cos(phi)]
        w = v[2] + self.U[:, :, None]
        f = -1 / (4 * self.d["Re"] * ek)
        return [self.spec(f * p) for p in (o[1] * w - o[2] * v[1], o[2] * v[0] - o[0] * w, o[0] * v[1] - o[1] * v[0])]

    def carreau_yasuda(self, u, v):
        rho, radius, mu0, muinf, lam, n, a = PLUGINS["carreau_yasuda"][1]
        lam = self.d["Re"] * lam * mu0 / (rho * radius ** 2)
        u = [u[0], u[1], u[2].clone()]
        u[2][:, 0] += self.U[:, 0]
        S = [[self.phys(self.D1 @ x) for x in u],
             [self.phys(x / self.r) for x in (1j * self.m * u[0] - u[1], 1j * self.m * u[1] + u[0], 1j * self.m * u[2])],
             [self.phys(1j * self.k * x) for x in u]]
        S = [[0.5 * (S[i][j] + S[j][i]) for j in range(3)] for i in range(3)]
        rate = torch.sqrt(2 * sum(S[i][j] ** 2 for i in range(3) for j in range(3)))
        e = muinf / mu0
        nu = e + (1 - e) * (1 + (lam * rate) ** a) ** (-n / a)
        g = [self.phys(x) for x in self.grad(self.spec(nu))]
        q = [self.phys(x) for x in self.curl(self.curl(u))]
        out = []
        for i in range(3):
            out.append(self.spec(((nu - 1) * -q[i] + 2 * sum(g[j] * S[j][i] for j in range(3))) / self.d["Re"]))
        return out

    def _diag(self, PM):
        d = -(self.m / self.r) ** 2 - self.k ** 2
        return d - (1 + 2 * PM * self.m) / self.r ** 2 if PM else d

    def _system(self, PM, BC, c1, c2):
        """LU factors of c1 + c2 Lap with the axis-parity and wall rows, per mode."""
        H = self.mi.numel()
        A = (c2 * self.lap).expand(H, -1, -1).clone()
        A.diagonal(dim1=1, dim2=2).add_((c2 * self._diag(PM) + c1).T)
        A[:, 0] = 0
        A[:, -1] = 0
        odd = ((self.m.round().long() + abs(PM)) % 2).bool()
        rows = [torch.tensor(x, device=DEV) for x in self.axis]
        A[:, 0, :KL + 1] = torch.where(odd[:, None], rows[0], rows[1])
        A[:, -1, -KL - 1:] = torch.tensor(self.wall[BC], device=DEV)
        if BC == 1:
            A[0] = torch.eye(self.N, dtype=torch.float64, device=DEV)
        return torch.linalg.lu_factor(A)

    def _solve(self, F, b, zero=False):
        """A x = b for complex (N, H) fields."""
        x = torch.linalg.lu_solve(*F, torch.view_as_real(b.T.contiguous()))
        x = torch.view_as_complex(x.contiguous()).T.clone()
        if zero:
            x[:, 0] = 0
        return x

    def _bc(self, up, um, uz):
        ur, ut = 0.5 * (up[-1] + um[-1]), -0.5j * (up[-1] - um[-1])
        dr = 0.5 * (self.wallz.to(up.dtype) @ (up[-KL - 1:] + um[-KL - 1:]))
        d = 1 / self.r[-1]
        return torch.stack([up[-1], um[-1], 1j * uz[-1],
                            ur * d + dr + 1j * d * self.m * ut + 1j * self.k * uz[-1]], -1)

    def matrices(self):
        d1, d2 = 1 / self.dt, -self.implicit / self.d["Re"]
        if self.LN is None:
            self.LN = self._system(0, 1, 0.0, 1.0)
        self.LD = [self._system(PM, 0, d1, d2) for PM in (1, -1, 0)]
        one = torch.zeros(self.N, self.mi.numel(), dtype=torch.complex128, device=DEV)
        one[-1] = 1
        nil = torch.zeros_like(one)
        a, b, c = (self._solve(F, one) for F in self.LD)
        g = self.grad(self._solve(self.LN, -one, zero=True))
        self.infl = [(a, nil, nil), (nil, b, nil), (nil, nil, 1j * c), (g[0] + 1j * g[1], g[0] - 1j * g[1], g[2])]
        B = torch.stack([self._bc(*x).real for x in self.infl], -1)  # (H, 4, 4)
        B[0] = torch.eye(4, dtype=torch.float64, device=DEV)
        self.Binv = torch.linalg.inv(B).to(torch.complex128)
        flux = torch.zeros(self.N, 1, dtype=torch.float64, device=DEV)
        flux[1:-1] = 1
        self.Ui = torch.linalg.lu_solve(self.LD[2][0][0], self.LD[2][1][0], flux)[:, 0]
        self.flux = 2 * (self.Ui @ self.w)

    def step(self, u0, N):
        d1, d2 = 1 / self.dt, (1 - self.implicit) / self.d["Re"]
        L = (d2 * self.lap).to(torch.complex128)
        rhs = []
        for PM, x, f in ((1, u0[0] + 1j * u0[1], N[0] + 1j * N[1]), (-1, u0[0] - 1j * u0[1], N[0] - 1j * N[1]),
                         (0, u0[2], N[2])):
            rhs.append(L @ x + (d2 * self._diag(PM) + d1) * x + f)
        r, t = 0.5 * (rhs[0] + rhs[1]), -0.5j * (rhs[0] - rhs[1])
        div = r / self.r + self.D1 @ r + 1j * self.m / self.r * t + 1j * self.k * rhs[2]
        div[0] = div[-1] = 0
        g = self.grad(self._solve(self.LN, div, zero=True))
        rhs = [rhs[0] - (g[0] + 1j * g[1]), rhs[1] - (g[0] - 1j * g[1]), rhs[2] - g[2]]
        for x in rhs:
            x[0] = x[-1] = 0
        x = [self._solve(F, b) for F, b in zip(self.LD, rhs)]
        a = -(self.Binv @ self._bc(*x)[:, :, None])[:, :, 0]
        a[0] = 0
        for i, c in enumerate(self.infl):
            # unit solutions are real (the axial ones imaginary): their real multiples carry Re and Im of a
            x = [y + a[:, i] * z for y, z in zip(x, c)]
        u = [0.5 * (x[0] + x[1]), -0.5j * (x[0] - x[1]), x[2]]
        u[2][:, 0] -= 2 * (u[2][:, 0].real @ self.w) / self.flux * self.Ui
        return self.sym(u)

    def correct(self, u, plugin):
        """One corrector pass; returns the new state and the size of the correction."""
        N = self.nonlinear(u, plugin)
        N = [self.implicit * x + (1 - self.implicit) * y for x, y in zip(N, self.N0)]
        new = self.step(self.u0, N)
        return new, max(float((x - y).abs().max()) for x, y in zip(u, new))

    def timestep(self, u, plugin="", orbit=False, adapt=None):
        self.u0 = self.sym(u)
        self.N0 = self.nonlinear(self.u0, plugin)
        if adapt is not None:
            adapt(self)
        u = self.step(self.u0, self.N0)
        it, last = 1, 1e99
        while True:
            u, err = self.correct(u, plugin)
            if it == 1:
                self.corr_dt = self.dt * math.sqrt(self.dterr / err)
            if orbit or plugin == "carreau_yasuda" or err > last or err <= self.dterr:
                break
            last, it = err, it + 1
        return u

    def cfl(self):
        r = self.r_np
        gap = np.diff(r)
        d = np.minimum(np.append(gap, gap[-1]), np.insert(gap, 0, gap[0]))
        mx = [x.abs().amax((1, 2)).cpu().numpy() for x in (self.v[0], self.v[1], self.v[2] + self.U[:, :, None])]
        return min((d / mx[0]).min(), (2 * math.pi / (3 * self.M * self.d["Mp"]) / mx[1]).min(),
                   (2 * math.pi / (self.d["alpha"] * 3 * self.K) / mx[2]).min())


# ------------------------------------------------------------------- the cases
def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _ok(status):
    if status != P._lib.PF_OK:
        raise RuntimeError(P.load().pf_last_error())


ONES = (C.c_double * 3)(1.0, 1.0, 1.0)
ADAPTIVE_DT0 = 0.004  # the first dt of the variable-dt runs, which may grow to the case's dt
SHIFT = (0.1, 0.2)    # the map's shifts back


def _host(u):
    return [(np.ascontiguousarray(x.real.cpu().numpy()), np.ascontiguousarray(x.imag.cpu().numpy())) for x in u]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "coll2phys":
        u = _Flow(case).seeded(seed, 1e-3)[:case["fields"]]
        return dict(kind=kind, dims=(case["N"], case["K"], case["M"]), lib=P.load(),
                    ins=[(x.real.T.contiguous(), x.imag.T.contiguous()) for x in u],
                    outs=[torch.empty(case["N"], 3 * case["M"], 3 * case["K"], dtype=torch.float64, device=DEV) for _ in u])
    if kind == "serve":
        reqs = []
        for i, d in enumerate(_mix(case)):
            reqs.append((_cfg(d), _nsteps(case, i), _host(_Flow(d).seeded(seed * 100 + i, case["energy"]))))
        return dict(kind=kind, server=P.Server(hbm_budget=40 * 10 ** 9), reqs=reqs)
    if kind == "batch":
        mix = _mix(case)
        b = P.Batch([_cfg(d) for d in mix])
        b.matrices()
        xs = [f.pack(f.seeded(seed * 100 + i, case["energy"])) for i, f in enumerate(map(_Flow, mix))]
        for p in b.pipes:
            _ok(p.lib.pf_orbit_set_scales(p.ctx, ONES, 1.0))
        return dict(kind=kind, batch=b, xs=xs, ys=[torch.zeros_like(x) for x in xs], steps=case["steps"])
    f = _Flow(case)
    x = f.pack(f.seeded(seed, case["energy"]))
    cfg = _cfg(case)
    if kind == "adaptive":
        cfg = _cfg(dict(case, dt=-1.0), maxdt=case["dt"])
    pipe = P.Pipe(cfg)
    if case["plugin"]:
        pipe.util_set(*PLUGINS[case["plugin"]])
    if kind == "map":
        x[0], x[1], x[2] = SHIFT[0], SHIFT[1], case["dt"] * case["steps"]
    orb = Orbit(pipe, [case["steps"]], [(0.0, 0.0, 1.0)])
    orb.set_scales([1.0, 1.0, 1.0], 1.0)
    if kind == "steps":
        pipe.vel_matrices()
    torch.cuda.synchronize()
    return dict(kind=kind, pipe=pipe, cfg=cfg, orb=orb, x=x, y=torch.zeros_like(x), steps=case["steps"])


def run(s):
    kind = s["kind"]
    if kind == "coll2phys":
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        for (re, im), out in zip(s["ins"], s["outs"]):
            _ok(s["lib"].pf_tra_coll2phys_noalloc(*s["dims"], _ptr(re), _ptr(im), _ptr(out), stream))
        return s["outs"]
    if kind == "serve":
        srv, reqs = s["server"], s["reqs"]
        late = max(1, len(reqs) * 2 // 5)
        ids = [srv.submit(*q) for q in reqs[:-late]]
        srv.step()
        ids += [srv.submit(*q) for q in reqs[-late:]]
        left = set(ids)
        while left:
            srv.step()
            left -= set(srv.finished())
        return [part for i in ids for field in srv.result(i) for part in field]
    if kind == "batch":
        b = s["batch"]
        for p, x in zip(b.pipes, s["xs"]):
            _ok(p.lib.pf_orbit_vec2rtz(p.ctx, _ptr(x)))
        b.step(s["steps"])
        for p, y in zip(b.pipes, s["ys"]):
            _ok(p.lib.pf_orbit_rtz2vec(p.ctx, _ptr(y)))
        return s["ys"]
    pipe, orb = s["pipe"], s["orb"]
    if kind == "map":
        orb.steporbit(s["steps"], s["x"], s["y"])
        return s["y"]
    if kind == "adaptive":
        pipe.reconfigure(s["cfg"])
        t = pipe.tim
        t.dt = ADAPTIVE_DT0
        pipe.set_tim(t)
        pipe.vel_matrices()
    orb.vec2rtz(s["x"])
    for _ in range(s["steps"]):
        pipe.timestep()
    orb.rtz2vec(s["y"])
    return (s["y"], pipe.tim.dt) if kind == "adaptive" else s["y"]


def _modes(d):
    return (2 * d["K"] - 1) * d["M"] - (d["K"] - 1)


def _step_work(d):
    """One timestep with one corrector pass: 36 passes over a field (main.f90:20-44 counted once each way), the
    transforms of two nonlinear evaluations and the banded solves of two half-steps."""
    Z, Th = 3 * d["K"], 3 * d["M"]
    fft = d["N"] * (9 * d["M"] * 5 * Z * math.log2(Z) + 4.5 * Z * 5 * Th * math.log2(Th))
    return 36 * 16 * d["N"] * _modes(d), 2 * fft + 2 * 2 * d["N"] * _modes(d) * (3 * 18 + 26 + 100)


def work(case):
    kind = case["kind"]
    if kind == "coll2phys":
        n, Z, Th = case["N"], 3 * case["K"], 3 * case["M"]
        return {"bytes": case["fields"] * (16.0 * n * _modes(case) + 8.0 * n * Z * Th),
                "flops": case["fields"] * n * (case["M"] * 5 * Z * math.log2(Z) + Z / 2 * 5 * Th * math.log2(Th))}
    bytes_ = flops = 0.0
    for i, d in enumerate(_mix(case) if kind in ("batch", "serve") else [case]):
        b, f = _step_work(d)
        n = _nsteps(case, i)
        bytes_ += n * b + 96.0 * d["N"] * _modes(d)  # the state in and out
        flops += n * f
        if kind in ("adaptive", "map", "serve"):  # four factor sets of 13 diagonals
            bytes_ += 4 * 13 * 8.0 * d["N"] * _modes(d)
            flops += 4 * 4 * 18.0 * d["N"] * _modes(d)
    return {"bytes": bytes_, "flops": flops}


def _adapter(state):
    """tim_new_tstep (timestep.f90:259-278): the dt rule of a variable-dt run."""
    def adapt(f):
        dt, cfl = min(f.dt * 1.11, f.d["dt"]), f.cfl()
        if state["step"] == 0:
            dt = min(dt, cfl * 0.1)
        dt = min(dt, cfl * 0.5)
        if state["step"] > 0:
            dt = min(dt, f.corr_dt * 0.95)
        state["wait"] -= 1
        grown = state["wait"] < 0
        if dt < f.dt * 0.95 or (dt > f.dt * 1.10 and grown) or (dt == f.d["dt"] and f.dt < dt and grown):
            if dt >= f.dt:
                state["wait"] = 99
            f.dt = dt
            f.matrices()
        state["step"] += 1
    return adapt


def exact(case, seed):
    kind = case["kind"]
    if kind == "coll2phys":
        f = _Flow(case)
        return [f.phys(x) for x in f.seeded(seed, 1e-3)[:case["fields"]]]
    if kind in ("batch", "serve"):
        out = []
        for i, d in enumerate(_mix(case)):
            f = _Flow(d)
            u = f.seeded(seed * 100 + i, case["energy"])
            f.matrices()
            for _ in range(_nsteps(case, i)):
                u = f.timestep(u, orbit=kind == "serve")
            out += [part for field in _host(u) for part in field] if kind == "serve" else [f.pack(u)]
            del f
        return out
    f = _Flow(case)
    u = f.seeded(seed, case["energy"])
    if kind == "adaptive":
        f.dt = ADAPTIVE_DT0
    f.matrices()
    adapt = _adapter({"step": 0, "wait": 0}) if kind == "adaptive" else None
    for _ in range(case["steps"]):
        u = f.timestep(u, case["plugin"], orbit=kind == "map", adapt=adapt)
    if kind == "map":
        turn = torch.exp(1j * (SHIFT[0] * f.m + SHIFT[1] * f.k))
        return f.pack([x * turn for x in u])
    return (f.pack(u), f.dt) if kind == "adaptive" else f.pack(u)

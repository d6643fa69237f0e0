"""Performance cases: the work that users of this library have it do, through its public entry points.

A case is one of five kinds:

  step      a resident cube advanced by Solver.step (the loop body: three sweeps, ghost wrap, dt,
            velocity splines, Heun advection), then its clock read, as the integration guide's loop
            does; with "stats" also the PrintStats line that the loop prints every ten steps
  plug      Solver.evolve(W, dt), the reference's GPU plug point: pinned host arrays in and out
  tracers   one step and the download of every particle (position and velocity in upload order),
            for a program that follows its particles
  output    one step, then what the loop forms at an output iteration: the particle property table,
            the particle statistics and the PrintStats line
  ensemble  many independent cubes advanced together by Ensemble.step

The sizes are those of the benchmark, the tests and the documents (16^3, 64^3, 256^3 with 10^6
particles, 512^3 with 4 x 10^6, the ensemble of 32 cubes), an odd grid, and generic ones.
"""
import math

import numpy as np
import torch

from dns_gkm_lpt_b200 import ic
from dns_gkm_lpt_b200.solver import Ensemble, Solver

F64 = torch.float64
GAM, RHO0, T0, R_GAS, PRANDTL = 1.4, 1.0, 300.0, 287.0, 0.70


def _case(name, kind, n, particles, Mt=0.3, Re=60.0, steps=1, stats=False, mixed=False, periodic=False,
          power_law=False, coef32=False, members=""):
    c = {"kind": kind, "n": n, "particles": particles, "Mt": Mt, "Re": Re, "steps": steps, "stats": stats,
         "mixed": mixed, "periodic": periodic, "power_law": power_law, "coef32": coef32, "members": members}
    return dict(c, name=name) if name else c


def listed():
    ens = "32x16 48x8 64x6 96x2"
    return [
        # a test-sized cube, one step at a time: launches and latency
        _case("cube_16", "step", 16, 64, Re=30.0),
        # the small production cube: ten steps and the statistics line the loop prints after them
        _case("cube_64_stats", "step", 64, 15625, Re=30.0, steps=10, stats=True),
        # an odd grid (no tensor copies), periodic splines and the power-law viscosity
        _case("cube_95_periodic", "step", 95, 20000, Mt=0.5, steps=4, periodic=True, power_law=True),
        # the headline cube in FP64 and in mixed precision
        _case("cube_256", "step", 256, 1000000),
        _case("cube_256_mixed", "step", 256, 1000000, mixed=True),
        # the large cube in FP64, and in the form that saves the most memory and time
        _case("cube_512", "step", 512, 4000000, Mt=0.5, Re=100.0),
        _case("cube_512_mixed", "step", 512, 4000000, Mt=0.5, Re=100.0, mixed=True, coef32=True),
        # the reference's own program on this library: host arrays in and out, every step
        _case("plug_256", "plug", 256, 0),
        # following particles: more particles than a step alone would need, read back after each
        _case("tracers_128", "tracers", 128, 1000000),
        # an output iteration
        _case("output_128", "output", 128, 100000),
        # a parameter study: cubes of uneven sizes stepped together, in both precisions
        _case("ensemble_32", "ensemble", 96, 10000, members=ens),
        _case("ensemble_32_mixed", "ensemble", 96, 10000, mixed=True, members=ens),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["plug", "tracers", "output", "ensemble"])
    Mt, Re = round(rng.uniform(0.1, 0.6), 3), round(rng.uniform(20.0, 100.0), 1)
    mixed = kind in ("step", "ensemble") and rng.random() < 0.4
    opts = {"Mt": Mt, "Re": Re, "mixed": mixed, "periodic": rng.random() < 0.3, "power_law": rng.random() < 0.3}
    if kind == "ensemble":
        sizes = sorted({_log_int(rng, 16, 96) for _ in range(rng.randint(2, 4))})
        members = " ".join("%dx%d" % (m, rng.randint(1, 8)) for m in sizes)
        return _case("", kind, sizes[-1], _log_int(rng, 500, 20000), members=members, **opts)
    if kind == "plug":
        return _case("", kind, _log_int(rng, 32, 200), 0, **opts)
    if kind == "step":
        n = _log_int(rng, 12, 400)
        return _case("", kind, n, _log_int(rng, 64, max(100, n ** 3 // 16)), steps=rng.randint(1, 8 if n <= 128 else 2),
                     stats=not mixed and rng.random() < 0.3, coef32=rng.random() < 0.25, **opts)
    n = _log_int(rng, 16, 160)
    return _case("", kind, n, _log_int(rng, 1000, 500000), **opts)


# ------------------------------------------------------------------- inputs --
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _field(n, Mt, Re, seed):
    """A turbulent field: solenoidal velocities with the initial-condition recipe's spectrum
    (k^4 exp(-2 (k/4)^2), 1 <= k <= 8) and smooth density and pressure fluctuations of order Mt^2,
    as a decaying field has them after its first steps.  Returns the parameters and the conserved
    interior state (5, n, n, n) in (y, x, z) order."""
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    kf = torch.fft.fftfreq(n, 1.0 / n, dtype=F64, device=dev)
    kr = torch.fft.rfftfreq(n, 1.0 / n, dtype=F64, device=dev)
    ky, kx, kz = kf.view(n, 1, 1), kf.view(1, n, 1), kr.view(1, 1, -1)
    ksq = ky * ky + kx * kx + kz * kz
    kk = ksq.sqrt()
    shell = (kk >= 1.0) & (kk <= min(8.0, n // 3))
    amp = torch.where(shell, kk * torch.exp(-((kk / 4.0) ** 2)), torch.zeros_like(kk))
    ksq = ksq.clamp_min(1e-14)

    def spectrum():
        return torch.fft.rfftn(torch.randn((n, n, n), generator=g, dtype=F64, device=dev)) * amp

    uh, vh, wh = spectrum(), spectrum(), spectrum()
    div = (uh * kx + vh * ky + wh * kz) / ksq
    u, v, w = (torch.fft.irfftn(h, s=(n, n, n)) for h in (uh - div * kx, vh - div * ky, wh - div * kz))
    del uh, vh, wh, div
    s1, s2 = (torch.fft.irfftn(spectrum(), s=(n, n, n)) for _ in range(2))
    s1 /= s1.std()
    s2 /= s2.std()
    p0 = RHO0 * R_GAS * T0
    fac = Mt * math.sqrt(GAM * p0 / RHO0) / float((u * u + v * v + w * w).mean().sqrt())
    u *= fac
    v *= fac
    w *= fac
    rho = RHO0 * (1.0 + 0.25 * Mt * Mt * s1)
    p = p0 * (1.0 + 0.25 * Mt * Mt * s2)
    dx = 2.0 * math.pi / n
    u2 = float((u * u + v * v + w * w).mean())
    sqdu = 0.0
    for a in (u, v, w):
        for ax in range(3):
            sqdu += float((((torch.roll(a, -1, ax) - torch.roll(a, 1, ax)) * (0.5 / dx)) ** 2).mean())
    P = ic.Params(n=n, gam=GAM, den0=RHO0, Mt=float(Mt), Re=float(Re), mu0=u2 * math.sqrt(5.0 / (3.0 * sqdu)) / Re,
                  p0=p0, t0=math.sqrt(5.0 * u2 / sqdu) / math.sqrt(u2 / 3.0))
    W = torch.stack([rho, rho * u, rho * v, rho * w, p / (GAM - 1.0) + 0.5 * rho * (u * u + v * v + w * w)])
    return P, W


def _wrap(W):
    """Interior state -> the reference layout with its three periodic ghost layers."""
    for ax in (1, 2, 3):
        n = W.shape[ax]
        idx = (torch.arange(-3, n + 3, device=W.device) % n)
        W = W.index_select(ax, idx)
    return W


def _positions(count, seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) + 7919)
    return (torch.rand((count, 3), generator=g, dtype=F64, device=_device()) * (2.0 * math.pi)).cpu().numpy()


def _members(case):
    out = []
    for part in case["members"].split():
        n, count = part.split("x")
        out += [int(n)] * int(count)
    return out


def _member_seed(seed, m):
    return int(seed) * 1009 + m


_CFL = 0.5


def prepare(case, seed):
    opts = {"cfl": _CFL, "visc_law": int(case["power_law"]), "spline_mode": int(case["periodic"])}
    if case["kind"] == "ensemble":
        specs = []
        for m, n in enumerate(_members(case)):
            P, W = _field(n, case["Mt"], case["Re"], _member_seed(seed, m))
            specs.append((P, _wrap(W), _positions(case["particles"], _member_seed(seed, m))))
        E = Ensemble([dict(opts, params=P, max_particles=case["particles"]) for P, _, _ in specs],
                     precision=int(case["mixed"]))
        for m, (_, W, pos) in enumerate(specs):
            E[m].upload_state(W)
            E[m].particles_upload(pos)
        E.autotune(2)
        return {"case": case, "E": E}
    P, W = _field(case["n"], case["Mt"], case["Re"], seed)
    s = Solver(P, max_particles=case["particles"], precision=int(case["mixed"]),
               spline_precision=int(case["coef32"]), **opts)
    W = _wrap(W)
    if case["kind"] == "plug":
        host = torch.empty(W.shape, dtype=F64, pin_memory=True)
        host.copy_(W)
        return {"case": case, "s": s, "W": host, "dt": float(_dt(W, P))}
    torch.cuda.synchronize()
    s.upload_state(W)
    s.synchronize()
    if case["particles"]:
        s.particles_upload(_positions(case["particles"], seed))
    return {"case": case, "s": s}


def _state_of(s, owner, mixed):
    """The state a program reads: the device view (kept with its owner), or, from the form that
    computes in single precision, the single-precision snapshot that holds all its digits."""
    W = s.device_state()
    if mixed:
        return W.float()
    W.owner = owner
    return W


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        E = state["E"]
        E.step(case["steps"])
        E.synchronize()
        return [_state_of(E[m], E, case["mixed"]) for m in range(len(E))]
    s = state["s"]
    if kind == "plug":
        s.evolve(state["W"], state["dt"])
        return state["W"]
    s.step(case["steps"])
    if kind == "tracers":
        pos, U = s.particles_download()
        return {"pos": pos, "U": U}
    if kind == "output":
        return {"particle_stats": s.particle_stats(), "props": s.particle_props(), "stats": s.print_stats()}
    out = {}
    if case["stats"]:
        out["stats"] = s.print_stats()
    t, dt, _ = s.clock()
    real = np.float32 if case["mixed"] else np.float64
    out.update(t=real(t), dt=real(dt), W=_state_of(s, s, case["mixed"]))
    return out


def work(case):
    """Per step of a cell: its state read and written once (80 B) and, for each of its three faces,
    five two-sided reconstructions and one flux, about 2,000 operations in all; per particle and
    step its position and velocity read and written (96 B) and two evaluations of three splines,
    about 800 operations; per spline coefficient its three line solves, 27 operations."""
    kind = case["kind"]
    sizes = _members(case) if kind == "ensemble" else [case["n"]]
    cells = sum(n ** 3 for n in sizes)
    parts = case["particles"] * len(sizes)
    b = case["steps"] * (80.0 * cells + 96.0 * parts)
    f = case["steps"] * (6000.0 * cells + (800.0 * parts + 81.0 * cells if parts else 0.0))
    if case["stats"] or kind == "output":
        b += 40.0 * cells
        f += 400.0 * cells
    if kind == "tracers":
        b += 48.0 * parts
    if kind == "output":   # five more splines, three Laplacians at the nodes, 41 values per particle
        b += 41 * 8.0 * parts
        f += (5 * 27 + 3 * 400) * cells + 8 * 600.0 * parts
    return {"bytes": b, "flops": f}


# ------------------------------------------- the same in 64 bits, with torch --
def _primitive(W):
    rho = W[0]
    u, v, w = W[1] / rho, W[2] / rho, W[3] / rho
    q = u * u + v * v + w * w
    p = (GAM - 1.0) * (W[4] - 0.5 * rho * q)
    return rho, u, v, w, q, p


def _dt(W, P):
    """cfl dx / max(|u| + c) over the interior of a state with ghosts."""
    rho, u, v, w, q, p = _primitive(W[:, 3:-3, 3:-3, 3:-3])
    return _CFL * P.dx / float((q.sqrt() + (GAM * p / rho).sqrt()).max())


def _weno(c):
    """Six cells -> the left and right values at the face between cells 2 and 3 (WENO-SYMOO)."""

    def side(a3, a2, a1, b1, b2, b3):
        P = (a3 / 3 - 7 * a2 / 6 + 11 * a1 / 6, -a2 / 6 + 5 * a1 / 6 + b1 / 3,
             a1 / 3 + 5 * b1 / 6 - b2 / 6, 11 * b1 / 6 - 7 * b2 / 6 + b3 / 3)
        S = [13.0 / 12 * (a3 - 2 * a2 + a1) ** 2 + 0.25 * (a3 - 4 * a2 + 3 * a1) ** 2,
             13.0 / 12 * (a2 - 2 * a1 + b1) ** 2 + 0.25 * (b1 - a2) ** 2,
             13.0 / 12 * (a1 - 2 * b1 + b2) ** 2 + 0.25 * (3 * a1 - 4 * b1 + b2) ** 2,
             13.0 / 12 * (b1 - 2 * b2 + b3) ** 2 + 0.25 * (5 * b1 - 8 * b2 + 3 * b3) ** 2]
        S[3] = torch.maximum(torch.maximum(S[0], S[1]), torch.maximum(S[2], S[3]))
        a = [g / (1e-10 + s) for g, s in zip((0.05, 0.45, 0.45, 0.05), S)]
        return (a[0] * P[0] + a[1] * P[1] + a[2] * P[2] + a[3] * P[3]) / (a[0] + a[1] + a[2] + a[3])

    return side(*c), side(*c[::-1])


class _Moments:
    """Moments of one Maxwellian: tables of <u^k> over all u and over one half space, <v^l>, <w^m>
    and <xi^2s>, and the vectors <u^k v^l w^m psi> and <u^k v^l w^m psi (psi . a)>."""

    def __init__(self, U, lam, K, half):
        s = 0.5 / lam
        self.full = []
        for x in U:
            t = [torch.ones_like(x), x]
            for i in range(2, 7):
                t.append(x * t[-1] + (i - 1) * s * t[-2])
            self.full.append(t)
        self.xi = (1.0, K * s, (K * K + 2 * K) * s * s)
        e = 0.5 * torch.exp(-lam * U[0] * U[0]) / (math.pi * lam).sqrt()
        self.pos = self._half(U[0], s, 0.5 * torch.erfc(-lam.sqrt() * U[0]), e)
        self.neg = self._half(U[0], s, 0.5 * torch.erfc(lam.sqrt() * U[0]), -e)
        self.N = {0: self.full[0], 1: self.pos, -1: self.neg}
        self.half = half

    @staticmethod
    def _half(u, s, h0, e):
        t = [h0, u * h0 + e]
        for i in range(2, 7):
            t.append(u * t[-1] + (i - 1) * s * t[-2])
        return t

    def m(self, tab, k, l, m, x=0):
        v = self.N[tab][k] * self.full[1][l] * self.full[2][m]
        return v if x == 0 else v * self.xi[x]

    def e4(self, tab, k, l, m, x=0):
        """<u^k v^l w^m xi^2x psi_4>"""
        return 0.5 * (self.m(tab, k + 2, l, m, x) + self.m(tab, k, l + 2, m, x) + self.m(tab, k, l, m + 2, x)
                      + self.m(tab, k, l, m, x + 1))

    def psi(self, tab, k, l=0, m=0):
        return [self.m(tab, k, l, m), self.m(tab, k + 1, l, m), self.m(tab, k, l + 1, m), self.m(tab, k, l, m + 1),
                self.e4(tab, k, l, m)]

    def psi_a(self, a, tab, k, l=0, m=0):
        out = []
        for d in ((0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)):
            p = self.psi(tab, k + d[0], l + d[1], m + d[2])
            out.append(a[0] * p[0] + a[1] * p[1] + a[2] * p[2] + a[3] * p[3] + a[4] * p[4])
        e44 = 0.5 * (self.e4(tab, k + 2, l, m) + self.e4(tab, k, l + 2, m) + self.e4(tab, k, l, m + 2)
                     + self.e4(tab, k, l, m, 1))
        out.append(a[0] * self.e4(tab, k, l, m) + a[1] * self.e4(tab, k + 1, l, m) + a[2] * self.e4(tab, k, l + 1, m)
                   + a[3] * self.e4(tab, k, l, m + 1) + a[4] * e44)
        return out


def _slopes(b, U, lam, K):
    q = U[0] ** 2 + U[1] ** 2 + U[2] ** 2 + (K + 3) / (2 * lam)
    r = [b[i + 1] - U[i] * b[0] for i in range(3)]
    a4 = (2 * b[4] - q * b[0] - 2 * (U[0] * r[0] + U[1] * r[1] + U[2] * r[2])) * 4 * lam * lam / ((K + 3) * PRANDTL)
    a = [2 * lam * r[i] - U[i] * a4 for i in range(3)]
    return [b[0] - a[0] * U[0] - a[1] * U[1] - a[2] * U[2] - 0.5 * a4 * q] + a + [a4]


def _prim_lam(W):
    rho, u, v, w, _, p = _primitive(W)
    return rho, (u, v, w), p, 0.5 * rho / p


def _flux(WL, WR, Wl, Wr, D, tau, dt, dx):
    """The gas-kinetic flux over [0, dt]; D: the normal, first and second tangential slopes (left, right)."""
    K = int((5.0 - 3.0 * GAM) / (GAM - 1.0))

    def add(*terms):
        return [sum(c * v[q] for c, v in terms) for q in range(5)]

    sides, We, by, bz = [], None, None, None
    for W, half, j in ((Wl, 1, 0), (Wr, -1, 1)):
        rho, U, p, lam = _prim_lam(W)
        M = _Moments(U, lam, K, half)
        a = [_slopes([d[j][q] / rho for q in range(5)], U, lam, K) for d in D]
        e, y, z = M.psi(half, 0), M.psi_a(a[1], half, 0), M.psi_a(a[2], half, 0)
        We = add((rho, e)) if We is None else add((1.0, We), (rho, e))
        by, bz = (y, z) if by is None else (add((1.0, by), (1.0, y)), add((1.0, bz), (1.0, z)))
        conv = add((-1.0, M.psi_a(a[0], 0, 1)), (-1.0, M.psi_a(a[1], 0, 0, 1)), (-1.0, M.psi_a(a[2], 0, 0, 0, 1)))
        sides.append((rho, U, p, lam, M, half, a, _slopes(conv, U, lam, K)))
    pl, pr = sides[0][2], sides[1][2]
    tau = tau + dt * (pl - pr).abs() / (pl + pr).abs()
    ex = torch.exp(-dt / tau)
    g0 = dt - tau * (1 - ex)
    g1 = -(1 - ex) / g0
    g2 = (-dt + 2 * tau * (1 - ex) - dt * ex) / g0
    g4 = (dt * ex - tau * (1 - ex)) / g0
    g5 = -tau * g1
    rho, U, _, lam = _prim_lam(We)
    E = _Moments(U, lam, K, 0)
    al = _slopes([2 * (We[q] - WL[q]) / (rho * dx) for q in range(5)], U, lam, K)
    ar = _slopes([2 * (WR[q] - We[q]) / (rho * dx) for q in range(5)], U, lam, K)
    ay, az = _slopes(by, U, lam, K), _slopes(bz, U, lam, K)
    B = add((g1 * rho, E.psi(0, 0)), (-g1, We), (g2 * rho, E.psi_a(al, 1, 1)), (g2 * rho, E.psi_a(ar, -1, 1)),
            (g2 * rho, E.psi_a(ay, 0, 0, 1)), (g2 * rho, E.psi_a(az, 0, 0, 0, 1)))
    Pc = tau * (1 - ex)
    Qc = -tau * dt * ex + tau * tau * (1 - ex)
    p0, p1, p2 = dt - Pc, 0.5 * dt * dt - tau * (dt - Pc), -tau * (dt - Pc) + Qc
    p4, p5 = -Qc - tau * Pc, -tau * Pc
    F = add((p0 * rho, E.psi(0, 1)), (p2 * rho, E.psi_a(al, 1, 2)), (p2 * rho, E.psi_a(ar, -1, 2)),
            (p2 * rho, E.psi_a(ay, 0, 1, 1)), (p2 * rho, E.psi_a(az, 0, 1, 0, 1)))
    for r, _, _, _, M, h, a, at in sides:
        G = add((1.0, M.psi_a(a[0], h, 1)), (1.0, M.psi_a(a[1], h, 0, 1)), (1.0, M.psi_a(a[2], h, 0, 0, 1)))
        B = add((1.0, B), ((g4 + g5) * r, G), (g5 * r, M.psi_a(at, h, 0)))
        G = add((1.0, M.psi_a(a[0], h, 2)), (1.0, M.psi_a(a[1], h, 1, 1)), (1.0, M.psi_a(a[2], h, 1, 0, 1)))
        F = add((1.0, F), (Pc * r, M.psi(h, 1)), (p4 * r, G), (p5 * r, M.psi_a(at, h, 1)))
    A = _slopes([x / rho for x in B], U, lam, K)
    return add((1.0, F), (p1 * rho, E.psi_a(A, 0, 1)))


# (normal axis, axis of the first tangential slope, of the second; momentum order of the face frame)
_SWEEPS = ((1, 0, 2, (0, 1, 2, 3, 4)), (0, 1, 2, (0, 2, 1, 3, 4)), (2, 1, 0, (0, 3, 2, 1, 4)))


def _sweep(W, P, dt, power_law, sweep):
    """Flux differences F(f) - F(f - 1) of one direction, (5, n, n, n) in (y, x, z) order."""
    ax, ay, az, order = sweep
    n, nt, dx = P.n, P.n + 6, P.dx
    V = W[list(order)].permute(0, 1 + ax, 1 + ay, 1 + az)
    out = torch.empty_like(W[:, 3:-3, 3:-3, 3:-3])
    dst = out[list(order)].permute(0, 1 + ax, 1 + ay, 1 + az).contiguous()
    step = max(1, 4_000_000 // (n * n))
    for c0 in range(0, n, step):
        c1 = min(n, c0 + step)
        S = V[:, :, c0 + 2:c1 + 4, 2:nt - 2]
        rho, _, _, _, _, p = _primitive(S)
        T = p / (rho * R_GAS)
        rec = [_weno([x[f:f + n + 1] for f in range(6)]) for x in (S[0], S[1], S[2], S[3], T)]
        face = []
        for j in range(2):
            r, a, b, c, Tf = (x[j] for x in rec)
            face.append([r, a, b, c, r * R_GAS * Tf / (GAM - 1.0) + 0.5 * (a * a + b * b + c * c) / r])
        mid = (slice(None), slice(1, -1), slice(1, -1))
        WL, WR = ([S[q][2 + j:n + 3 + j][mid] for q in range(5)] for j in range(2))
        D = [[], [], []]
        for j in range(2):
            x = face[j]
            D[0].append([(2 * (x[q][mid] - WL[q]) if j == 0 else 2 * (WR[q] - x[q][mid])) / dx for q in range(5)])
            D[1].append([0.5 * (x[q][:, 2:, 1:-1] - x[q][:, :-2, 1:-1]) / dx for q in range(5)])
            D[2].append([0.5 * (x[q][:, 1:-1, 2:] - x[q][:, 1:-1, :-2]) / dx for q in range(5)])
        pL, TL = p[2:n + 3][mid], T[2:n + 3][mid]
        x = TL / P.T0
        mu = P.mu0 * x ** 0.76 if power_law else P.mu0 * x ** 1.5 * (P.T0 + 110.4) / (TL + 110.4)
        F = _flux(WL, WR, [y[mid] for y in face[0]], [y[mid] for y in face[1]], D, mu / pL, dt, dx)
        for q in range(5):
            dst[q][:, c0:c1] = F[q][1:] - F[q][:-1]
    inv = [order.index(q) for q in range(5)]
    axes = (ax, ay, az)
    return dst[inv].permute(0, *(1 + axes.index(i) for i in range(3)))


def _eulerian(W, P, dt, power_law):
    acc = sum(_sweep(W, P, dt, power_law, s) for s in _SWEEPS)
    return _wrap(W[:, 3:-3, 3:-3, 3:-3] - acc / P.dx)


class _Splines:
    """Uniform tricubic B-splines of arrays on the spline grid, by dense line solves."""

    def __init__(self, P, periodic):
        n, dx, dev = P.n, P.dx, _device()
        self.periodic, self.h = periodic, dx
        self.N = n if periodic else n + 6
        self.x0 = 0.5 * dx - (0.0 if periodic else 3 * dx)
        N = self.N
        if periodic:
            A = torch.zeros((N, N), dtype=F64, device=dev)
            i = torch.arange(N, device=dev)
            for o, c in ((-1, 1.0), (0, 4.0), (1, 1.0)):
                A[i, (i + o) % N] += c / 6.0
            B = torch.linalg.inv(A)
            self.B = B[torch.arange(-1, N + 2, device=dev) % N]
        else:
            A = torch.zeros((N + 2, N + 2), dtype=F64, device=dev)
            i = torch.arange(N, device=dev)
            for o, c in ((0, 1.0), (1, 4.0), (2, 1.0)):
                A[1 + i, i + o] = c / 6.0
            for r, at in ((0, 0), (N + 1, N - 1)):
                A[r, at], A[r, at + 1], A[r, at + 2] = 1.0, -2.0, 1.0
            self.B = torch.linalg.inv(A)[:, 1:N + 1]

    def coefs(self, f):
        for ax in range(3):
            f = torch.tensordot(self.B, f, ([1], [ax])).movedim(0, ax)
        return f.contiguous()

    def nodes(self, W, fn):
        return fn(W[:, 3:-3, 3:-3, 3:-3] if self.periodic else W)

    def _basis(self, x):
        t = (x - self.x0) / self.h
        i = torch.floor(t)
        if not self.periodic:
            i = i.clamp(0, self.N - 2)
        t = t - i
        s = 1.0 - t
        w = (s ** 3 / 6, (3 * t ** 3 - 6 * t ** 2 + 4) / 6, (-3 * t ** 3 + 3 * t ** 2 + 3 * t + 1) / 6, t ** 3 / 6)
        d = tuple(c / self.h for c in (-0.5 * s * s, 1.5 * t * t - 2 * t, -1.5 * t * t + t + 0.5, 0.5 * t * t))
        h = tuple(c / self.h ** 2 for c in (s, 3 * t - 2, -3 * t + 1, t))
        i = i.long()
        return (i % self.N if self.periodic else i), (w, d, h)

    def at(self, C, pos, orders):
        """Derivatives of the spline C at positions (count, 3): one result per (a, b, c) of orders."""
        M = C.shape[0]
        (ia, A), (ib, B), (ic_, Z) = (self._basis(pos[:, k]) for k in range(3))
        flat, out = C.reshape(-1), [0.0] * len(orders)
        for x in range(4):
            for y in range(4):
                for z in range(4):
                    c = flat[((ia + x) * M + ib + y) * M + ic_ + z]
                    for k, (p, q, r) in enumerate(orders):
                        out[k] = out[k] + A[p][x] * B[q][y] * Z[r][z] * c
        return out

    def at_nodes(self, C, orders, off):
        """The same at the n^3 nodes whose coefficient windows start at off."""
        n = C.shape[0] - 2 * off - (3 if self.periodic else 2)
        w = ((1 / 6.0, 4 / 6.0, 1 / 6.0), (-0.5 / self.h, 0.0, 0.5 / self.h),
             (1 / self.h ** 2, -2 / self.h ** 2, 1 / self.h ** 2))
        out = []
        for o in orders:
            f = C
            for ax in range(3):
                f = sum(w[o[ax]][x] * f.narrow(ax, off + x, n) for x in range(3))
            out.append(f)
        return out


_GRAD = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
_VALUE = ((0, 0, 0),)


def _velocity_splines(W, P, periodic, coef32=False):
    S = _Splines(P, periodic)
    C = [S.coefs(S.nodes(W, lambda V, q=q: V[q] / V[0])) for q in (1, 2, 3)]
    return S, [c.float().double() for c in C] if coef32 else C


def _heun(S, C, pos, U, dt):
    swap = [1, 0, 2]   # positions are (y, x, z), velocities (u, v, w)
    U2 = torch.stack([S.at(c, pos + U[:, swap] * dt, _VALUE)[0] for c in C], 1)
    pos = pos + (0.5 * (U + U2) * dt)[:, swap]
    pos = torch.where(pos > 2 * math.pi, pos - 2 * math.pi, pos)
    pos = torch.where(pos < 0, pos + 2 * math.pi, pos)
    return pos, torch.stack([S.at(c, pos, _VALUE)[0] for c in C], 1)


def _print_stats(W, P, periodic, power_law, t, coef32=False):
    S, C = _velocity_splines(W, P, periodic, coef32)
    rho, u, v, w, q, p = _primitive(W[:, 3:-3, 3:-3, 3:-3])
    T = p / (rho * R_GAS)
    g = [S.at_nodes(c, _GRAD, 0 if periodic else 3) for c in C]   # [u, v, w][d/dy, d/dx, d/dz]
    x = T / P.T0
    mu = P.mu0 * x ** 0.76 if power_law else P.mu0 * x ** 1.5 * (P.T0 + 110.4) / (T + 110.4)
    (uy, ux, uz), (vy, vx, vz), (wy, wx, wz) = g
    sij = (ux ** 2 + vy ** 2 + wz ** 2 + 0.5 * (uy + vx) ** 2 + 0.5 * (uz + wx) ** 2 + 0.5 * (wy + vz) ** 2).mean()
    out = {"t_over_t0": t / P.t0, "TKE": (rho * q).mean(), "Diss": (mu * sum(d * d for a in g for d in a)).mean(),
           "SijSij": sij}
    for name, d in (("u", ux), ("v", vy), ("w", wz)):
        m2 = (d ** 2).mean()
        out["SKEW" + name] = (d ** 3).mean() / m2 ** 1.5
        out["KURT" + name] = (d ** 4).mean() / m2 ** 2
    for name, f, scale in (("Prms", p, GAM * P.p0 * P.Mt ** 2), ("Trms", T, (GAM - 1) * P.T0 * P.Mt ** 2),
                           ("Vrms", 1 / rho, P.Mt ** 2 / P.den0)):
        out[name] = ((f - f.mean()) ** 2).mean().sqrt() / scale
    return {k: float(x) for k, x in out.items()}


def _particle_table(W, P, periodic, pos):
    S, C = _velocity_splines(W, P, periodic)
    n, off = P.n, 0 if periodic else 3
    lap = []
    for c in C:
        nodes = torch.zeros((S.N,) * 3, dtype=F64, device=W.device)
        nodes[off:off + n, off:off + n, off:off + n] = sum(
            S.at_nodes(c, ((2, 0, 0), (0, 2, 0), (0, 0, 2)), off))
        lap.append(S.coefs(nodes))
    value_grad = _VALUE + _GRAD
    hess = ((2, 0, 0), (1, 1, 0), (1, 0, 1), (1, 1, 0), (0, 2, 0), (0, 1, 1), (1, 0, 1), (0, 1, 1), (0, 0, 2))

    def many(c, orders):
        return [torch.cat(x) for x in zip(*(S.at(c, pos[i:i + 100000], orders) for i in range(0, len(pos), 100000)))]

    rho = many(S.coefs(S.nodes(W, lambda V: V[0])), value_grad)
    vel = [many(c, value_grad) for c in C]
    prs = many(S.coefs(S.nodes(W, lambda V: _primitive(V)[5])), value_grad + hess)
    laps = [many(c, value_grad) for c in lap]
    cols = rho + [v[0] for v in vel] + [d for v in vel for d in v[1:]] + prs
    cols += [v[0] for v in laps] + [d for v in laps for d in v[1:]]
    (uy, ux, uz), (vy, vx, vz), (wy, wx, wz) = (v[1:] for v in vel)
    sij = ux ** 2 + vy ** 2 + wz ** 2 + 0.5 * (uy + vx) ** 2 + 0.5 * (uz + wx) ** 2 + 0.5 * (wy + vz) ** 2
    stats = {"TKE": sum(v[0] ** 2 for v in vel).mean(), "SijSij": sij.mean(),
             "SKEWu": (ux ** 3).mean() / (ux ** 2).mean() ** 1.5, "SKEWw": (wz ** 3).mean() / (wz ** 2).mean() ** 1.5}
    return torch.stack(cols, 1), {**{k: float(x) for k, x in stats.items()}, "count": None}


def exact(case, seed):
    if case["kind"] == "ensemble":
        out = []
        for m, n in enumerate(_members(case)):
            P, W = _field(n, case["Mt"], case["Re"], _member_seed(seed, m))
            W = _wrap(W)
            for _ in range(case["steps"]):
                W = _eulerian(W, P, _dt(W, P), case["power_law"])
            out.append(W)
        return out
    P, W = _field(case["n"], case["Mt"], case["Re"], seed)
    W = _wrap(W)
    if case["kind"] == "plug":
        return _eulerian(W, P, _dt(W, P), case["power_law"]).cpu()
    follow = case["kind"] in ("tracers", "output")
    if follow:
        pos = torch.from_numpy(_positions(case["particles"], seed)).to(W.device)
        S, C = _velocity_splines(W, P, case["periodic"])
        U = torch.stack([S.at(c, pos, _VALUE)[0] for c in C], 1)
        del C
    t, dt = 0.0, _dt(W, P)
    for _ in range(case["steps"]):
        W = _eulerian(W, P, dt, case["power_law"])
        if follow:
            S, C = _velocity_splines(W, P, case["periodic"])
            pos, U = _heun(S, C, pos, U, dt)
            del C
        last, dt = dt, _dt(W, P)
        t += dt
    if case["kind"] == "tracers":
        return {"pos": pos, "U": U}
    if case["kind"] == "output":
        table, ps = _particle_table(W, P, case["periodic"], pos)
        return {"particle_stats": ps, "props": table,
                "stats": _print_stats(W, P, case["periodic"], case["power_law"], t)}
    out = {"t": t, "dt": last, "W": W}
    if case["stats"]:
        out["stats"] = _print_stats(W, P, case["periodic"], case["power_law"], t, case["coef32"])
    return out

"""Measured cases of the phase-field framework.

A pass (`run`) is what a program of this framework does between two of its
outputs: a block of time steps on a resident state, then the state read back
(Tecplot output of the reference's program: phi, T, c; checkpoints: DPP too)
and, where the program monitors its run, the diagnostics and the tracking.
Everything goes through the package's public entry points (`pf3d.Domain`,
`pf3d.Batch`, `pf3d.karma.Karma`).

The states are those of a run under way, made from a seed: a solid with
columnar tips growing into the melt, the equilibrium interface profile, the
solute boundary layer ahead of it and slow composition waves everywhere else
(Karma model: a four-fold crystal in a supersaturated melt).

`exact` restates both models in 64-bit torch, without the package.
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "phase-field-project-3d_b200"))

import pf3d  # noqa: E402
from pf3d import deck, karma  # noqa: E402


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def domain(name, nx, ny, nz, precision, steps, **over):
    """One domain of the Al-Cu model.  path: "step" (the fused time loop),
    "probed" (one step at a time with the two-cell progress read of the
    reference's program), "monitored" (diagnostics and tracking every 4
    steps), "subroutines" (the reference's subroutines called one by one)."""
    c = {"name": name, "kind": "domain", "nx": nx, "ny": ny, "nz": nz, "precision": precision, "steps": steps,
         "path": "step", "dx": 0.5e-6, "quintic": 0, "noise": 0, "sweeps": 2, "T0": 917.0, "AAA": 0.01}
    c.update(over)
    return c


def crystal(name, nx, ny, nz, precision, steps, Fnoise):
    """One domain of the Karma model (karma3d.f90)."""
    return {"name": name, "kind": "karma", "nx": nx, "ny": ny, "nz": nz, "precision": precision, "steps": steps,
            "Fnoise": Fnoise}


def listed():
    return [
        # interactive use and the smallest domains: every step is followed by
        # the two-cell progress print of equacao_campo_fase.f90:174
        domain("tiny_fp64_probed", 36, 32, 48, 64, 20, path="probed"),
        # the 64 x 64 x 128 configuration, the size parity runs use
        domain("c1_fp64", 64, 64, 128, 64, 200),
        # the deck reader's defaults (quintic h, smooth noise, one sweep) on a
        # grid no dimension of which fits the tiles
        domain("ragged_defaults_fp64", 97, 131, 201, 64, 80, quintic=1, noise=2, sweeps=1),
        # the reference's documented production run: 340 x 340 x 700 at 0.15 um
        domain("run6_fp64", 340, 340, 700, 64, 50, dx=0.15e-6, AAA=0.03),
        # FP32: an ordinary odd-sized domain with the zero-mean noise
        domain("ragged_fp32", 150, 111, 190, 32, 200, noise=1),
        # FP32: the 256 x 256 x 512 replica of the 1024^3 configuration
        domain("replica_fp32", 256, 256, 512, 32, 150),
        # a run that logs energies, solute balance, solid fraction and tip
        domain("monitored_fp32", 192, 192, 384, 32, 80, path="monitored"),
        # the Fortran program's drop-in: one call per subroutine
        domain("subroutines_fp64", 128, 128, 256, 64, 12, path="subroutines"),
        # uneven domains stepped together in a server's quanta
        {"name": "batch_fp32", "kind": "batch", "domains": 12, "xmin": 32, "xmax": 128, "zmax": 256, "precision": 32,
         "steps": 320, "quantum": 16, "sizes": 3},
        # the Karma program's default domain with its noise (run3)
        crystal("karma_run3_fp64", 200, 200, 200, 64, 300, 0.01),
        crystal("karma_fp32", 256, 256, 256, 32, 200, 0.01),
        # a small Karma domain, without noise (the program's default)
        crystal("karma_small_fp64", 72, 60, 80, 64, 300, 0.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["domain", "domain", "domain", "domain", "batch", "karma", "karma"])
    prec = rng.choice([64, 32])
    if kind == "batch":
        return {"kind": "batch", "domains": rng.randint(2, 14), "xmin": 32, "xmax": _log(rng, 48, 128),
                "zmax": _log(rng, 128, 256), "precision": prec, "steps": rng.randint(4, 16) * 16, "quantum": 16,
                "sizes": rng.randrange(1 << 20)}
    if kind == "karma":
        c = crystal("", *(_log(rng, 40, 256) for _ in range(3)), prec, rng.randint(100, 250), rng.choice([0.0, 0.01]))
        del c["name"]
        return c
    while True:
        nx, ny, nz = _log(rng, 24, 340), _log(rng, 24, 340), _log(rng, 32, 700)
        if nx * ny * nz <= 30e6:
            break
    path = rng.choice(["step", "step", "step", "step", "probed", "monitored", "subroutines"])
    cells = nx * ny * nz
    steps = rng.randint(30, 200) if path in ("step", "monitored") else rng.randint(8, 24)
    if path == "monitored":
        steps = steps // 4 * 4
    if cells > 8e6:
        steps = min(steps, 60)
    c = domain("", nx, ny, nz, prec, steps, path=path, quintic=rng.choice([0, 0, 1]), noise=rng.choice([0, 0, 1, 2]),
               sweeps=rng.choice([2, 2, 2, 1, 3]), dx=rng.choice([0.5e-6, 0.15e-6]), T0=round(rng.uniform(915, 919), 3),
               AAA=round(rng.uniform(0.0, 0.02), 4))
    del c["name"]
    return c


def batch_sizes(case):
    rng = random.Random(case["sizes"])
    got = []
    for _ in range(case["domains"]):
        x = _log(rng, case["xmin"], case["xmax"])
        got.append((x, x, _log(rng, x, case["zmax"]), rng.uniform(915.0, 919.0), rng.uniform(0.0, 0.02)))
    return got


def work(case):
    """Each step reads and writes every state field of every cell once (Al-Cu:
    phi, c, T, DPP; Karma: phi, U).  Operations per cell and step: the two
    sweeps and the solute update of the Al-Cu model (621 floating-point
    operations as counted on the device), the two passes of the Karma model."""
    es = case["precision"] // 8
    if case["kind"] == "batch":
        cells = sum(x * y * z for x, y, z, _, _ in batch_sizes(case))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    n = cells * case["steps"]
    if case["kind"] == "karma":
        return {"bytes": n * 4 * es, "flops": n * 450}
    sweeps = case.get("sweeps", 2)
    return {"bytes": n * 8 * es, "flops": n * (230 * sweeps + 160)}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _axes(nx, ny, nz):
    a = [torch.arange(n, dtype=torch.float64, device="cuda") for n in (nz, ny, nx)]
    return a[0][:, None, None], a[1][None, :, None], a[2][None, None, :]


def _waves(nx, ny, nz, g, amplitude):
    """Slow waves of a few periods across the domain."""
    k, j, i = _axes(nx, ny, nz)
    f = torch.rand(4, 3, generator=g, device="cuda", dtype=torch.float64) * 3 + 0.5
    ph = torch.rand(4, generator=g, device="cuda", dtype=torch.float64) * 6.28
    s = torch.zeros(nz, ny, nx, dtype=torch.float64, device="cuda")
    for q in range(4):
        s += torch.sin(6.2831853 * (f[q, 0] * k / nz + f[q, 1] * j / ny + f[q, 2] * i / nx) + ph[q])
    return s.mul_(amplitude / 4)


def melt_state(nx, ny, nz, T0, precision, g):
    """A columnar front under way: phi, c, T, DPP in 64 bits (values that are
    representable in the case's precision)."""
    k, j, i = _axes(nx, ny, nz)
    r = torch.rand(24, 4, generator=g, device="cuda", dtype=torch.float64)
    H = torch.full((1, ny, nx), 0.3 * nz, dtype=torch.float64, device="cuda") + (r[0, 0] - 0.5) * 4
    for q in range(24):   # tips of different heights
        rad = 5 + 9 * r[q, 3]
        H = H + 0.25 * nz * r[q, 2] * torch.exp(-((i - r[q, 0] * nx) ** 2 + (j - r[q, 1] * ny) ** 2) / (rad * rad))
    H = torch.clamp(H, max=0.8 * nz)
    gy, gx = torch.gradient(H[0])
    d = (k - H) / torch.sqrt(1 + gx * gx + gy * gy)[None]   # signed distance to the front, cells
    phi = 1.0 / (1.0 + torch.exp(torch.clamp(d, max=700.0)))   # (1 - tanh(d/2))/2: width 4 cells
    ke = float(np.float32(0.14))
    cl = 0.0196 + ((933.3 - T0) / 640.0 - 0.0196) * torch.exp(-torch.clamp(d, min=0.0) / 12.0)
    c = cl * (1.0 - (1.0 - ke) * phi) * (1.0 + _waves(nx, ny, nz, g, 0.02))
    del cl, d
    dpp = 1e-3 * phi * (1.0 - phi)
    T = T0 + _waves(nx, ny, nz, g, 0.05)
    st = {"phi": phi, "c": c, "T": T, "dpp": dpp}
    if precision == 32:
        st = {n: v.float().double() for n, v in st.items()}
    return st


def crystal_state(nx, ny, nz, dx, omega, precision, g):
    """A four-fold crystal at the corner and its diffusion layer: phi, U."""
    k, j, i = _axes(nx, ny, nz)
    x, y, z = (i + 0.5) * dx, (j + 0.5) * dx, (k + 0.5) * dx
    u = torch.rand(4, generator=g, device="cuda", dtype=torch.float64)
    r = torch.sqrt(x * x + y * y + z * z)
    s4 = (x ** 4 + y ** 4 + z ** 4) / r ** 4
    R = dx * min(nx, ny, nz) * (0.35 + 0.15 * u[0]) * (1 + (0.3 + 0.2 * u[1]) * (s4 - 0.6))
    d = r - R
    phi = -torch.tanh(d / math.sqrt(2.0))
    U = -omega * (1 - torch.exp(-torch.clamp(d, min=0.0) / (6 + 6 * u[2]))) * (1.0 + _waves(nx, ny, nz, g, 0.02))
    st = {"phi": phi, "U": U}
    if precision == 32:
        st = {n: v.float().double() for n, v in st.items()}
    return st


def _params(case, T0=None, AAA=None):
    return deck.run6_params(T0=case["T0"] if T0 is None else T0, taxa_resfr=19.84,
                            AAA=case["AAA"] if AAA is None else AAA, h_quintico=case.get("quintic", 0),
                            ruido_tipo=case.get("noise", 0), n_varreduras=case.get("sweeps", 2))


NAMES = {"phi": "phase_field_old", "c": "conc_soluto_old", "T": "TOLD", "dpp": "DPP"}


def prepare(case, seed):
    """What the program holds before the block: the resident domain with its
    state, and pinned host buffers for the fields it reads back."""
    torch.cuda.synchronize()
    g = _gen(seed)
    s = dict(case)
    if case["kind"] == "karma":
        p = karma.karma_params(nx=case["nx"], ny=case["ny"], nz=case["nz"], Fnoise=case["Fnoise"])
        st = crystal_state(p.nx, p.ny, p.nz, p.dx, karma.derived(p).Omega, case["precision"], g)
        k = karma.Karma(p, case["precision"])
        k.upload(st["phi"].cpu().numpy(), st["U"].cpu().numpy())
        s["karma"] = k
        return s
    if case["kind"] == "batch":
        b = pf3d.Batch(case["precision"])
        s["slots"] = []
        for n, (nx, ny, nz, T0, AAA) in enumerate(batch_sizes(case)):
            slot = b.add(deck.grid(nx, ny, nz, 0.5e-6), _params({}, T0, AAA))
            st = melt_state(nx, ny, nz, T0, case["precision"], g)
            b.load_state(slot, {n: v.cpu().numpy() for n, v in st.items()})
            s["slots"].append(slot)
        s["batch"] = b
        return s
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    d = pf3d.Domain(deck.grid(nx, ny, nz, case["dx"]), _params(case), case["precision"])
    st = melt_state(nx, ny, nz, case["T0"], case["precision"], g)
    host = {n: torch.empty(nz, ny, nx, dtype=torch.float64, pin_memory=True) for n in NAMES}
    for n, name in NAMES.items():
        host[n].copy_(st[n])
        d.upload(name, host[n].numpy())
    s["domain"], s["host"] = d, host
    if case["precision"] == 32:   # an FP32 program keeps FP32 snapshots
        s["snap"] = {n: torch.empty(nz, ny, nx, dtype=torch.float32) for n in ("phi", "c", "T")}
    return s


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(s):
    return {"karma": run_karma, "batch": run_batch, "domain": run_domain}[s["kind"]](s)


def read_back(s):
    d, host = s["domain"], s["host"]
    if s["precision"] == 64:
        for n, name in NAMES.items():
            d.download(name, host[n].numpy())
        return dict(host)
    for n in ("phi", "c", "T"):   # what the program's output holds
        d.download(NAMES[n], host[n].numpy())
        s["snap"][n].copy_(host[n])
    return dict(s["snap"])


def run_domain(s):
    d, n, path = s["domain"], s["steps"], s["path"]
    if path == "probed":
        seen = []
        for _ in range(n):
            d.step(1)
            seen.append(d.probe("phase_field_old", s["nx"] // 2, 10, s["nz"] // 2))
            seen.append(d.probe("phase_field_old", s["nx"] // 2, min(100, s["ny"] - 1), s["nz"] // 2))
        out = read_back(s)
        out["seen"] = np.array(seen, dtype=np.float64 if s["precision"] == 64 else np.float32)
        return out
    if path == "monitored":
        log, tip = [], []
        for _ in range(n // 4):
            log.append(d.step_diag(4))
            tip.append(d.track()[:2])
        out = read_back(s)
        kind = np.float64 if s["precision"] == 64 else np.float32
        out["log"], out["tip"] = np.array(log, dtype=kind), np.array(tip, dtype=kind)
        return out
    if path == "subroutines":
        d.step_reference_order(n)
    else:
        d.step(n)
    return read_back(s)


def run_batch(s):
    b = s["batch"]
    for _ in range(s["steps"] // s["quantum"]):   # a server's loop
        b.step_async(s["quantum"])
        b.wait()
        b.progress()
    kind = np.float64 if s["precision"] == 64 else np.float32
    out = {"log": np.array([b.diagnosticos(q) for q in s["slots"]], dtype=kind),
           "tip": np.array([b.track(q)[:2] for q in s["slots"]], dtype=kind)}
    for f in ("phi", "c", "T"):
        out[f] = [b.download(q, NAMES[f]).astype(kind, copy=False) for q in s["slots"]]
    return out


def run_karma(s):
    k = s["karma"]
    k.step(s["steps"])
    kind = np.float64 if s["precision"] == 64 else np.float32
    out = {n: k.download(f).astype(kind, copy=False) for n, f in (("phi", 0), ("U", 1))}
    out["tip"] = np.array(k.tip(), dtype=np.float64)
    return out


# --------------------------------------------------------------------------
# the same in 64-bit torch
# --------------------------------------------------------------------------
def exact(case, seed):
    g = _gen(seed)
    if case["kind"] == "karma":
        return exact_karma(case, g)
    if case["kind"] == "batch":
        out = {"log": [], "tip": None, "phi": [], "c": [], "T": []}
        for nx, ny, nz, T0, AAA in batch_sizes(case):
            m = AlCu(nx, ny, nz, dict(case, dx=0.5e-6, T0=T0, AAA=AAA, quintic=0, noise=0, sweeps=2),
                     melt_state(nx, ny, nz, T0, case["precision"], g))
            for _ in range(case["steps"]):
                m.step()
            out["log"].append(m.diagnostics())
            for f in ("phi", "c", "T"):
                out[f].append(getattr(m, f).cpu())
        out["log"] = np.array(out["log"])
        return out
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    m = AlCu(nx, ny, nz, case, melt_state(nx, ny, nz, case["T0"], case["precision"], g))
    seen, log = [], []
    for n in range(case["steps"]):
        m.step()
        if case["path"] == "probed":
            for y in (10, min(100, ny - 1)):
                seen.append(float(m.phi[nz // 2 - 1, y - 1, nx // 2 - 1]))
        if case["path"] == "monitored" and n % 4 == 3:
            log.append(m.diagnostics())
    out = {n: getattr(m, n) for n in (("phi", "c", "T", "dpp") if case["precision"] == 64 else ("phi", "c", "T"))}
    if case["path"] == "probed":
        out["seen"] = np.array(seen)
    if case["path"] == "monitored":
        out["log"], out["tip"] = np.array(log), None
    return out


def _i64(v):
    return v - (1 << 64) if v >= 1 << 63 else v


def _hash(i, j, k, it, salt, device="cuda"):
    """The reference's integer noise, in [0, 1): h is taken modulo 2**64."""
    h = i * 2654435761 + j * 2246822519 + k * 3266489917 + (it * 668265263 + salt * 374761393 + 1)
    for m in (0xff51afd7ed558ccd, 0xc4ceb9fe1a85ec53, None):
        h = h ^ ((h >> 33) & 0x7fffffff)
        if m is not None:
            h = h * _i64(m)
    return (h & 0x7fffffffffffffff).double() * 2.0 ** -63


class AlCu:
    """The coupled Al-Cu step (principal.f90:93-226), array sections in 64 bits."""

    def __init__(self, nx, ny, nz, case, st):
        self.n = (nx, ny, nz)
        self.dx = dx = case["dx"]
        self.hq, self.rt, self.sweeps = case["quintic"], case["noise"], case["sweeps"]
        f4 = lambda v: float(np.float32(v))  # noqa: E731
        self.Ke, sigma, self.ajuste = f4(0.14), f4(0.093), 2.0
        self.Tm, self.T0, self.rate, self.Me, self.Vm, self.R = 933.3, case["T0"], 19.84, 640.0, 1.130e-05, 8.31451
        self.DE, self.Dl, self.Ds, self.dH_cp = 0.03, 3.0e-09, 3.0e-13, 0.891002e9 / 2.926560e+06
        self.sigma = sigma
        self.dt = dx * dx / (7.5 * self.Dl)
        ratio = self.dt / (dx * dx / (5.0 * self.Dl))
        self.AAA = case["AAA"] * (ratio if self.rt == 0 else math.sqrt(ratio))
        # W0, E0: the fixed-point scan of W0_E0.f90:10-31
        inc, k1 = f4(1e-7), 1.5556349186104 / (4.0 * dx)
        a = f4(np.float32(2.0) * np.float32(0.093)) * 4.24264068711929
        e = np.cumsum(np.concatenate([[0.0], np.full(200000, inc)]))
        with np.errstate(divide="ignore"):
            E = a / np.sqrt((k1 * e) ** 2)
        q = int(np.argmax(np.abs(E - e) < 1e-5))
        self.W0, self.E0 = float((k1 * e[q]) ** 2), float(E[q])
        self.TP, self.M0, self.it = self.T0, 1.9e-03, 0
        self.phi, self.c, self.T, self.dpp = (st[n] for n in ("phi", "c", "T", "dpp"))

    def mobility(self, cs, cl):
        """auxiliar.f90:12-42"""
        total, ph = 0.0, 0.11
        while True:
            hp = ph * ph * (3.0 - 2.0 * ph)
            total += hp * (1 - hp) / (((1 - hp) * cl * (1 - cl) + hp * cs * (1 - cs)) * ph * (1 - ph))
            ph += 0.01
            if ph > 0.8999:
                break
        f4 = lambda v: float(np.float32(v))  # noqa: E731
        integral = f4(0.01) / 2 * (f4(54.39180136) + 2 * total + 234.073053)
        qsi = self.R * self.TP / self.Vm * (cl - cs) ** 2 * integral
        kin = self.R * self.TP * f4(np.float32(1) - np.float32(0.14)) / (self.Vm * self.Me)
        return self.ajuste / (self.E0 ** 2 / self.sigma * (kin + self.E0 * qsi / (self.Dl * math.sqrt(2 * self.W0))))

    def noise(self):
        nx, ny, nz = self.n
        i, j, k = (torch.arange(3, n - 1, device="cuda") for n in (nx, ny, nz))
        if self.rt != 2:
            return _hash(i[None, None, :], j[None, :, None], k[:, None, None], self.it, 1).float().double()
        L = [torch.arange(n // 6 + 2, device="cuda") for n in (nx, ny, nz)]
        lat = _hash(L[0][None, None, :], L[1][None, :, None], L[2][:, None, None], self.it // 20, 3)
        for axis, q in ((2, i), (1, j), (0, k)):   # trilinear, x first
            f = ((q % 6).double() / 6.0).reshape([-1 if a == axis else 1 for a in range(3)])
            lat = (1 - f) * lat.index_select(axis, q // 6) + f * lat.index_select(axis, q // 6 + 1)
        return lat.float().double()

    def sweep(self, cs, cl):
        nx, ny, nz = self.n
        p, dx = self.phi, self.dx

        def P(a, b, e):
            return p[2 + e:nz - 2 + e, 2 + b:ny - 2 + b, 2 + a:nx - 2 + a]

        h = 0.5 / dx
        g = [(p[1:-1, 1:-1, 2:] - p[1:-1, 1:-1, :-2]) * h, (p[1:-1, 2:, 1:-1] - p[1:-1, :-2, 1:-1]) * h,
             (p[2:, 1:-1, 1:-1] - p[:-2, 1:-1, 1:-1]) * h]
        s = [v * v for v in g]
        Q2 = (s[0] + s[1] + s[2] + 1e-23).square_()
        eps = self.E0 * (1 + self.DE * (4 * (s[0] * s[0] + s[1] * s[1] + s[2] * s[2]) / Q2 - 3))
        f = 16 * self.E0 * self.DE * eps / Q2
        ex = [f * g[a] * g[b] * (s[a] - s[b]) for a, b in ((0, 1), (1, 2), (2, 0))]   # exy, eyz, ezx
        del f, Q2, s, g
        eps.square_()
        at = {"E": (1, 0, 0), "W": (-1, 0, 0), "N": (0, 1, 0), "S": (0, -1, 0), "T": (0, 0, 1), "B": (0, 0, -1)}

        def node(v, n):
            a, b, e = at[n]
            return v[1 + e:nz - 3 + e, 1 + b:ny - 3 + b, 1 + a:nx - 3 + a]

        PP = P(0, 0, 0)
        AA = torch.zeros_like(PP)
        for n in at:
            AA += node(eps, n) * (P(*at[n]) - PP)
        AA /= dx * dx
        # the cross terms: each pair of axes (u, v) with its coefficient
        for e, U, V in ((ex[0], ("E", "W"), ("N", "S")), (ex[1], ("N", "S"), ("T", "B")), (ex[2], ("T", "B"), ("E", "W"))):
            (up, um), (vp, vm) = U, V
            add = lambda *ns: tuple(sum(at[q][r] for q in ns) for r in range(3))  # noqa: E731
            acc = node(e, up) * (P(*add(up, vp)) - P(*add(up, vm)) + P(*at[vp]) - P(*at[vm]))
            acc += node(e, vp) * (P(*add(um, vp)) - P(*add(up, vp)) + P(*at[um]) - P(*at[up]))
            acc += node(e, um) * (P(*add(um, vm)) - P(*add(um, vp)) + P(*at[vm]) - P(*at[vp]))
            acc += node(e, vm) * (P(*add(up, vm)) - P(*add(um, vm)) + P(*at[up]) - P(*at[um]))
            AA += (0.25 / (dx * dx)) * acc
        del ex, eps, acc
        q = 1 - PP
        if self.hq:
            hl, hh = 30 * PP * PP * q * q, PP ** 3 * (10 - 15 * PP + 6 * PP * PP)
        else:
            hl, hh = 6 * PP * q, PP * PP * (3 - 2 * PP)
        C = self.c[2:nz - 2, 2:ny - 2, 2:nx - 2]
        den = self.Ke * hh + (1 - hh)
        arg = ((1 - cs) * (1 - C / den) / ((1 - cl) * (1 - self.Ke * C / den))).abs_()
        AA += self.R * self.TP / self.Vm * hl * torch.log(arg) - self.W0 * 2 * PP * q * (1 - 2 * PP)
        r = self.noise()
        if self.rt != 0:
            r = 2 * r - 1
        new = PP + self.M0 * self.dt * AA + r * self.AAA * 16 * PP * PP * q * q
        self.dpp = self.dpp.clone()
        self.dpp[2:-2, 2:-2, 2:-2] = new - PP
        pn = p.clone()
        pn[2:-2, 2:-2, 2:-2] = torch.clamp(new, 0.0, 1.0)
        for axis in (1, 2, 0):   # equacao_campo_fase.f90:151-167
            for to, of in ((0, 1), (1, 2), (-1, -2), (-2, -3)):
                pn.select(axis, to).copy_(pn.select(axis, of))
        return pn

    def solute(self):
        p, c = self.phi, self.c
        h = p ** 3 * (10 - 15 * p + 6 * p * p) if self.hq else p * p * (3 - 2 * p)
        den = self.Ke * h + (1 - h)
        CL = c / den
        CS = self.Ke * CL
        G = (1 - h) * CL * (1 - CL) + h * CS * (1 - CS)
        mu = torch.log(CL / (1 - CL))
        del h, den, CL, CS
        inner = (slice(1, -1),) * 3
        D = torch.full_like(p[inner], self.Dl).masked_fill_(p[inner] > 0.95, self.Ds)
        GP, muP = G[inner], mu[inner]
        acc = torch.zeros_like(GP)
        for axis in range(3):
            for sl in (slice(2, None), slice(0, -2)):
                at = tuple(sl if a == axis else slice(1, -1) for a in range(3))
                acc += 2 * GP * G[at] / (GP + G[at]) * (mu[at] - muP)
        cn = c.clone()
        cn[inner] += acc * D * (self.dt / (self.dx * self.dx))
        co = cn.clone()
        for axis in (1, 2, 0):   # concentracao_soluto.f90:116-124
            cn.select(axis, 0).copy_(co.select(axis, 1))
            cn.select(axis, -1).copy_(co.select(axis, -2))
        return cn

    def step(self):
        self.it += 1
        inner = (slice(1, -1),) * 3
        P = self.phi[inner]
        hl = 30 * P * P * (1 - P) * (1 - P) if self.hq else 2 * P * (3 - 2 * P) - 2 * P * P
        self.T = self.T.clone()
        self.T[inner] = self.dH_cp * hl * self.dpp[inner] + self.TP   # D = 0
        self.TP = self.T0 - self.rate * self.dt * self.it
        cs, cl = (self.Tm - self.TP) * self.Ke / self.Me, (self.Tm - self.TP) / self.Me
        new = self.sweep(cs, cl)
        for _ in range(self.sweeps - 1):
            self.phi = new
            new = self.sweep(cs, cl)
        self.c = self.solute()
        self.phi = new
        self.M0 = self.mobility(cs, cl)

    def diagnostics(self):
        p, dx = self.phi, self.dx
        grad2 = torch.zeros_like(p)
        grad2[1:-1, 1:-1, 1:-1] = ((p[1:-1, 1:-1, 2:] - p[1:-1, 1:-1, :-2]) ** 2
                                   + (p[1:-1, 2:, 1:-1] - p[1:-1, :-2, 1:-1]) ** 2
                                   + (p[2:, 1:-1, 1:-1] - p[:-2, 1:-1, 1:-1]) ** 2) * (0.5 / dx) ** 2
        fe = (0.5 * self.E0 ** 2 * grad2 + self.W0 * p * p * (1 - p) * (1 - p)) * dx ** 3
        return (math.sqrt(float((p * p).sum())), float(p.max()), float(p.min()), float(self.c.sum()), float(fe.sum()))


def exact_karma(case, g):
    """karma3d.f90:160-287 on ghost-padded arrays."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dx, dt, e4, lam, kk, Fn = 0.8, 0.008, 0.02, 4.0, 0.14, case["Fnoise"]
    cl0 = (933.3 - 909.5) / 640.0
    st = crystal_state(nx, ny, nz, dx, (cl0 - 0.0196) / ((1.0 - kk) * cl0), case["precision"], g)
    D, at, om3 = 0.6267 * lam, 1 / (2 * math.sqrt(2.0)), 1.0 - 3.0 * e4
    idx = 1.0 / dx
    q = 0.25 * idx

    def ghost(v):
        return torch.nn.functional.pad(v[None, None], (1,) * 6, mode="replicate")[0, 0]

    def S(v, o):
        return v[1 + o[2]:nz + 1 + o[2], 1 + o[1]:ny + 1 + o[1], 1 + o[0]:nx + 1 + o[0]]

    def gradients(p, axis, sign):
        """the gradient at the face in direction sign * axis, axis by axis"""
        e = [0, 0, 0]
        e[axis] = sign
        got = []
        for a in range(3):
            if a == axis:
                got.append((S(p, e) - S(p, (0, 0, 0))) * (idx * sign))
                continue
            u = [0, 0, 0]
            u[a] = 1
            w = [-v for v in u]
            both = lambda s, t: tuple(x + y for x, y in zip(s, t))  # noqa: E731
            got.append(q * (S(p, u) + S(p, both(u, e)) - S(p, w) - S(p, both(w, e))))
        return got, e

    i, j, k = (torch.arange(1, n + 1, device="cuda") for n in (nx, ny, nz))
    phi, U = st["phi"], st["U"]
    for it in range(1, case["steps"] + 1):
        p, u = ghost(phi), ghost(U)
        div = torch.zeros_like(phi)
        for axis in range(3):
            for sign in (1, -1):
                gr, _ = gradients(p, axis, sign)
                gs = gr[0] * gr[0] + gr[1] * gr[1] + gr[2] * gr[2]
                small = gs < 1e-20
                gs = torch.where(small, 1.0, gs)
                s4 = gr[0] ** 4 + gr[1] ** 4 + gr[2] ** 4
                a_s = om3 + 4 * e4 * s4 / (gs * gs)
                J = a_s * (a_s * gr[axis] + 16 * e4 * (gr[axis] ** 3 - gr[axis] * s4 / gs) / gs)
                div += sign * torch.where(small, om3 * om3 * gr[axis], J)
        c = [0.5 * idx * (S(p, tuple(int(a == b) for b in range(3))) - S(p, tuple(-int(a == b) for b in range(3))))
             for a in range(3)]
        gm = c[0] * c[0] + c[1] * c[1] + c[2] * c[2]
        big = gm > 1e-20
        s4 = (c[0] ** 4 + c[1] ** 4 + c[2] ** 4) / torch.where(big, gm * gm, 1.0)
        as2 = torch.where(big, (om3 + 4 * e4 * s4) ** 2, om3 * om3)
        om = 1 - phi * phi
        d = (div * idx + phi - phi ** 3 - lam * om * om * U) / as2
        if Fn != 0.0:
            h = _hash(i[None, None, :], j[None, :, None], k[:, None, None], it, 0)
            d += Fn * (2 * h - 1) * om / math.sqrt(dt)
        dg = ghost(d)
        rhs = torch.zeros_like(U)
        cell = (1 + (1 - kk) * U) * d
        for axis in range(3):
            for sign in (1, -1):
                gr, e = gradients(p, axis, sign)
                gmag = torch.sqrt(gr[0] * gr[0] + gr[1] * gr[1] + gr[2] * gr[2])
                F = D * 0.25 * (2 - phi - S(p, e)) * (S(u, e) - U) * (sign * idx)
                cf = 0.5 * (cell + (1 + (1 - kk) * S(u, e)) * S(dg, e))
                F += torch.where(gmag > 1e-10, at * cf * gr[axis] / torch.where(gmag > 1e-10, gmag, 1.0), 0.0)
                rhs += sign * F
        rhs = rhs * idx + 0.5 * cell
        U = U + dt * rhs / (0.5 * (1 + kk) - 0.5 * (1 - kk) * phi)
        phi = torch.clamp(phi + dt * d, -1.0, 1.0)
    ax = (phi[0, 0, :] > 0).nonzero().flatten()
    n = min(nx, ny, nz)
    r = torch.arange(n, device="cuda")
    dg = (phi[r, r, r] > 0).nonzero().flatten()
    tip = [float(v[-1] + 1) if len(v) else 0.0 for v in (ax, dg)]
    return {"phi": phi, "U": U, "tip": np.array(tip)}

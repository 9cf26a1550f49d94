"""Workloads of the MD step engine, each called as a user's program calls it.

A case is a dict of plain values. `kind` says which calls a pass makes:

  run      Verlet.run_host: positions and velocities in from page-locked
           buffers, `steps` velocity-Verlet steps (the Verlet list rebuilt on
           the half-skin rule), positions, velocities and forces back
  lists    VerletList.update and .csr: a neighbour analysis of one frame
  sample   energies, virials and totals of one frame, with the per-atom records
  serve    a batch of independent small systems through Server

`system` names the atoms: argon (fcc, LJsCut), copper (fcc, EAM), nial (B2 with
vacancies, Multi with three EAM tables), liquid (LJ argon at liquid density).
Units are nm, ps, g/mol, kJ/mol.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import mdcraft_gb300 as mdg

EV = 96.48533212331
KB = 0.008314462175
SIGMA, EPS, AR_MASS = 0.3405, 0.0104 * EV, 39.948
CU_MASS, NI_MASS, AL_MASS = 63.546, 58.6934, 26.9815
LJ_RC = 2.5 * SIGMA
TAU = SIGMA * math.sqrt(AR_MASS / EPS)
CU_RC, NIAL_RC, EAM_SKIN = 0.5, 0.6, 0.05
NIAL = {(0, 0): (0.25, 8.0, 0.249), (1, 1): (0.15, 9.0, 0.286), (0, 1): (0.20, 8.5, 0.250)}

# lattice constant, rc, skin, dt, temperature
SYSTEMS = {
    "argon": dict(a=0.526, rc=LJ_RC, skin=0.03, dt=0.002, T=100.0),
    "copper": dict(a=0.3615, rc=CU_RC, skin=EAM_SKIN, dt=0.001, T=300.0),
    "nial": dict(a=0.288, rc=NIAL_RC, skin=EAM_SKIN, dt=0.001, T=600.0),
    "liquid": dict(a=(4.0 / 0.8442) ** (1.0 / 3.0) * SIGMA, rc=LJ_RC, skin=0.3 * SIGMA, dt=0.005 * TAU,
                   T=0.72 * EPS / KB),
}


def _case(name, kind, system, cells, precision="mixed", steps=0, nvt=False, requests=0, n_max=0):
    c = dict(kind=kind, system=system, nx=cells[0], ny=cells[1], nz=cells[2], precision=precision, steps=steps,
             nvt=nvt, requests=requests, n_max=n_max)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a host program that moves 500 atoms one step at a time, in the reference's arithmetic
        _case("argon 500 fp64 one step", "run", "argon", (5, 5, 5), "fp64", 1),
        # the plain LJ run of the benchmark's first configuration, in both arithmetics
        _case("argon 4000 fp64", "run", "argon", (10, 10, 10), "fp64", 25),
        _case("argon 4000 mixed", "run", "argon", (10, 10, 10), "mixed", 100),
        # an equilibration at constant temperature of a mid-sized, not quite cubic crystal
        _case("copper 32k mixed nvt", "run", "copper", (19, 20, 21), "mixed", 50, nvt=True),
        # the headline configuration: a production run, the same run driven from the host a step at a time, and the
        # reference's arithmetic
        _case("copper 1M mixed", "run", "copper", (63, 63, 63), "mixed", 25),
        _case("copper 1M mixed one step", "run", "copper", (63, 63, 63), "mixed", 1),
        _case("copper 1M fp64", "run", "copper", (63, 63, 63), "fp64", 2),
        # the two-species alloy
        _case("nial 1M mixed", "run", "nial", (80, 80, 80), "mixed", 10),
        # a large liquid, whose list is rebuilt every seven or eight steps
        _case("liquid 4M mixed", "run", "liquid", (100, 100, 100), "mixed", 15),
        # neighbours of every atom of a frame (coordination, pair distribution)
        _case("lists 62k", "lists", "argon", (25, 25, 25)),
        # the thermodynamic sample a production run takes every few hundred steps
        _case("sample copper 108k", "sample", "copper", (30, 30, 30)),
        # a screening batch: independent small systems of both kinds
        _case("serve 48", "serve", "", (0, 0, 0), "mixed", 100, requests=48, n_max=8192),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _cells(rng, atoms, per_cell, least):
    """Near-cubic cell counts of about `atoms` atoms, each edge by itself, none under `least`."""
    c = (atoms / per_cell) ** (1.0 / 3.0)
    return tuple(max(least, int(round(c * rng.uniform(0.85, 1.18)))) for _ in range(3))


def draw(rng):
    what = rng.choice(["small", "small", "mid", "mid", "fp64", "alloy", "large", "lists", "sample", "serve"])
    if what == "small":  # one-step calls and short runs of the smallest systems
        steps = rng.choice([1, rng.randint(20, 100)])
        system = rng.choice(["argon", "copper"])
        return _case("", "run", system, _cells(rng, _log_uniform(rng, 500, 8000), 4, 4), rng.choice(["fp64", "mixed"]),
                     min(steps, 30) if steps > 1 else 1)
    if what == "mid":
        system = rng.choice(["argon", "copper", "liquid"])
        return _case("", "run", system, _cells(rng, _log_uniform(rng, 8000, 250000), 4, 8), "mixed",
                     rng.choice([1, rng.randint(10, 50)]), nvt=rng.random() < 0.3)
    if what == "fp64":
        system = rng.choice(["argon", "copper", "liquid"])
        return _case("", "run", system, _cells(rng, _log_uniform(rng, 8000, 500000), 4, 8), "fp64", rng.randint(1, 3),
                     nvt=rng.random() < 0.3)
    if what == "alloy":
        return _case("", "run", "nial", _cells(rng, _log_uniform(rng, 4000, 600000), 2, 6),
                     rng.choice(["mixed", "mixed", "fp64"]), rng.randint(1, 4))
    if what == "large":
        system = rng.choice(["copper", "liquid"])
        return _case("", "run", system, _cells(rng, _log_uniform(rng, 250000, 1500000), 4, 8), "mixed",
                     rng.randint(1, 20))
    if what == "lists":
        return _case("", "lists", rng.choice(["argon", "copper"]),
                     _cells(rng, _log_uniform(rng, 1000, 80000), 4, 5))
    if what == "sample":
        return _case("", "sample", rng.choice(["argon", "copper", "nial"]),
                     _cells(rng, _log_uniform(rng, 2000, 150000), 3, 6), rng.choice(["mixed", "fp64"]))
    return _case("", "serve", "", (0, 0, 0), "mixed", rng.randint(20, 100), requests=rng.randint(4, 64),
                 n_max=int(_log_uniform(rng, 1024, 8192)))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _sites(nx, ny, nz, a, basis):
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    cells = np.stack([x.ravel(), y.ravel(), z.ravel()], 1).astype(np.float64)
    return ((cells[:, None, :] + np.asarray(basis)[None]) * a).reshape(-1, 3) + 0.25 * a


FCC = [[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]]
B2 = [[0, 0, 0], [0.5, 0.5, 0.5]]


def _inputs(system, nx, ny, nz, seed, jitter=0.01):
    """Positions, velocities, masses, kinds and box edges of one system: a lattice inside its periodic box with small
    random displacements, Maxwell-Boltzmann velocities and a slow drift of the whole."""
    p = SYSTEMS[system]
    rng = np.random.default_rng(seed)
    a = p["a"]
    L = np.array([nx * a, ny * a, nz * a])
    r = _sites(nx, ny, nz, a, B2 if system == "nial" else FCC)
    kind = np.zeros(len(r), dtype=np.uint16)
    if system == "nial":  # Ni on the corners, Al on the centres, one site in 200 vacant
        kind[1::2] = 1
        keep = np.sort(rng.permutation(len(r))[len(r) // 200:])
        r, kind = r[keep], kind[keep]
        m = np.where(kind == 0, NI_MASS, AL_MASS)
    else:
        m = np.full(len(r), CU_MASS if system == "copper" else AR_MASS)
    if system == "liquid":  # bounded, so that no pair of millions starts on top of another
        r += rng.uniform(-0.05 * a, 0.05 * a, size=r.shape)
    else:
        r += rng.standard_normal(r.shape) * (jitter * a if system != "nial" else 0.003 * a)
    r = np.mod(r, L)
    r = np.where(r >= L, r - L, r)
    v = rng.standard_normal(r.shape) * np.sqrt(KB * p["T"] / m)[:, None]
    v -= (m[:, None] * v).sum(0) / m.sum()
    v += np.array([0.01, -0.02, 0.015])
    return r, v, m, kind, L


def _tables(A, p, re, rc, rho_max, nr=5000, nrho=5000):
    """Finnis-Sinclair-type tables: rho(r), r phi(r) and F(rho) on uniform grids from zero."""
    dr, drh = rc * 1.1 / (nr - 1), rho_max / (nrho - 1)
    r = np.arange(nr) * dr
    return dict(rc=rc, F=-np.sqrt(np.arange(nrho) * drh) * EV, R=np.exp(-3.0 * (r / re - 1.0)),
                V=r * A * np.exp(-p * (r / re - 1.0)) * EV, nr=nr, dr=dr, nrho=nrho, drh=drh)


def _tables_of(system):
    """The EAM tables by kind pair."""
    if system == "copper":
        return {(0, 0): _tables(0.2, 9.0, 0.2556, CU_RC, 33.0)}
    return {k: _tables(A, p, re, NIAL_RC, 80.0) for k, (A, p, re) in NIAL.items()}


def _records(r, v, m, kind, p):
    at = mdg.new_atoms(len(r))
    at["r"], at["v"], at["m"], at["kind"] = r, v, m, kind
    at["rcut"], at["rns"] = p["rc"], p["rc"] + p["skin"]
    at["uid"] = np.arange(1, len(r) + 1)
    return at


def _domain(L):
    d = mdg.Domain(0.0, L[0], 0.0, L[1], 0.0, L[2])
    for k in range(3):
        d.set_periodic(k, True)
    return d


def _eam(t):
    return mdg.EAM(t["rc"], t["F"], t["R"], t["V"], t["nr"], t["dr"], t["nrho"], t["drh"])


def _solver(system, precision):
    if system in ("argon", "liquid"):
        return mdg.Single(mdg.LJsCut(EPS, SIGMA, LJ_RC), periodic=True, precision=precision)
    tabs = _tables_of(system)
    if system == "copper":
        return mdg.Single(_eam(tabs[0, 0]), periodic=True, precision=precision)
    s = mdg.Multi(2, periodic=True, precision=precision)
    for (i, j), t in tabs.items():
        s.add_potential(i, j, _eam(t))
    return s


_kept = {}


def _context():
    """One context for the whole program, as a user's program has it."""
    if "ctx" not in _kept:
        _kept["ctx"] = mdg.Context(0)
    return _kept["ctx"]


def _pinned(a):
    """A page-locked copy of a host array."""
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
    t[...] = a
    return t


NVT = dict(beta=2.0, seed=77)


def _served(case, seed):
    """The requests of one batch: (system, nx, ny, nz, seed), sizes log-uniform from 256 atoms, three in five argon.
    The batch's sizes are the case's own; the atoms are the seed's."""
    rng = np.random.default_rng(case["requests"] * 100003 + case["n_max"])
    out = []
    for k in range(case["requests"]):
        system = "argon" if rng.random() < 0.6 else "copper"
        p = SYSTEMS[system]
        least = int(math.ceil(2.0 * (p["rc"] + p["skin"]) / p["a"]))
        c = math.exp(rng.uniform(math.log(256), math.log(case["n_max"]))) / 4.0
        nx = max(least, int(round(c ** (1.0 / 3.0))))
        ny = max(least, int(round(math.sqrt(c / nx))))
        out.append((system, nx, ny, max(least, int(round(c / (nx * ny)))), seed * 1009 + k))
    return out


def prepare(case, seed):
    if case["kind"] == "serve":
        # one server for the whole program: requests come and go
        if "server" not in _kept:
            _kept["server"] = mdg.Server(slots=64, max_atoms=16384, order="balanced")
            _kept["solvers"] = {s: _solver(s, "mixed") for s in ("argon", "copper")}
        reqs = []
        for system, nx, ny, nz, sd in _served(case, seed):
            r, v, m, kind, L = _inputs(system, nx, ny, nz, sd)
            reqs.append((system, _records(r, v, m, kind, SYSTEMS[system]), _domain(L)))
        return dict(kind="serve", server=_kept["server"], solvers=_kept["solvers"], reqs=reqs, steps=case["steps"])
    p = SYSTEMS[case["system"]]
    # a cold frame for the neighbour analysis, its atoms in no order: its shells stand apart, and every frame has as
    # many neighbours
    frame = case["kind"] == "lists"
    r, v, m, kind, L = _inputs(case["system"], case["nx"], case["ny"], case["nz"], seed, 0.004 if frame else 0.01)
    if frame:
        r = r[np.random.default_rng(seed).permutation(len(r))]
    atoms = _records(r, v, m, kind, p)
    st = dict(kind=case["kind"], sys=mdg.System(_context(), _domain(L), atoms), steps=case["steps"], dt=p["dt"])
    st["list"] = mdg.VerletList(st["sys"])
    if case["kind"] == "lists":
        return st
    st["list"].update()
    s = st["solver"] = _solver(case["system"], case["precision"])
    if case["nvt"]:
        s.set_thermostat(mdg.Langevin(NVT["beta"], p["T"], p["dt"], seed=NVT["seed"]))
    s.prepare(st["sys"])
    s.stages(st["sys"])
    if case["kind"] == "sample":
        st["records"] = atoms
        return st
    st["verlet"] = mdg.Verlet(s)
    st["pos"], st["vel"], st["force"] = _pinned(r), _pinned(v), _pinned(np.zeros_like(r))
    return st


def run(state):
    if state["kind"] == "run":
        state["verlet"].run_host(state["sys"], state["dt"], state["steps"], state["pos"], state["vel"], state["force"])
        return {"r": state["pos"], "v": state["vel"], "f": state["force"]}
    if state["kind"] == "lists":
        state["list"].update()
        first, neighbours = state["list"].csr()
        return {"first": first.view(np.int64), "neighbours": neighbours.view(np.int64)}
    if state["kind"] == "sample":
        state["solver"].virials(state["sys"])
        totals = state["sys"].measure()
        at = state["sys"].download(state["records"])
        return {"Ep": at["Ep"], "Em": at["Em"], "V": at["V"], "totals": totals}
    server, solvers = state["server"], state["solvers"]
    ids = [server.submit(solvers[s], dom, at, SYSTEMS[s]["dt"], state["steps"]) for s, at, dom in state["reqs"]]
    done = []
    for i in ids:
        server.wait(i, 120.0)
        at, info = server.result(i)
        if info["status"] != 0:
            raise RuntimeError("request %d ended with status %d" % (i, info["status"]))
        done.append(at)
    return {k: np.concatenate([at[k] for at in done]) for k in ("r", "v", "f")}


# ---------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------
def _per_atom(system):
    """Atoms per unit cell, pairs within the cutoff and listed pairs per atom, operations per atom and step."""
    p = SYSTEMS[system]
    per_cell = 2 if system == "nial" else 4
    density = per_cell / p["a"] ** 3
    pairs = 4.0 / 3.0 * math.pi * p["rc"] ** 3 * density
    listed_pairs = 4.0 / 3.0 * math.pi * (p["rc"] + p["skin"]) ** 3 * density
    # distance 8, LJ force 11 + 6; EAM: distance, r and interval 14, density cubic 7, force 22
    ops = 25.0 * pairs if system in ("argon", "liquid") else (21.0 + 36.0) * pairs
    return per_cell, pairs, listed_pairs, ops + 30.0


def work(case):
    if case["kind"] == "serve":
        b = f = 0.0
        for system, nx, ny, nz, _ in _served(case, 1):
            _, _, lp, ops = _per_atom(system)
            n = 4.0 * nx * ny * nz
            b += n * 2 * 208 + case["steps"] * n * (96.0 + 4.0 * lp)
            f += case["steps"] * n * ops
        return {"bytes": b, "flops": f}
    per_cell, pairs, lp, ops = _per_atom(case["system"])
    n = float(per_cell * case["nx"] * case["ny"] * case["nz"])
    if case["kind"] == "lists":  # positions in, lists out; each candidate sphere tested once
        return {"bytes": n * (24.0 + 8.0 + 8.0 * (lp + 1.0)), "flops": n * 9.0 * lp}
    if case["kind"] == "sample":  # state and list in, Ep, Em, V out
        return {"bytes": n * (56.0 + 4.0 * lp + 88.0), "flops": n * (ops + 20.0 * pairs)}
    # inputs and outputs of the call; per step the state read and written and the list read
    return {"bytes": n * 120.0 + case["steps"] * n * (96.0 + 4.0 * lp), "flops": case["steps"] * n * ops}


# ---------------------------------------------------------------------------
# the same results in 64 bits, with plain torch
# ---------------------------------------------------------------------------
_dev = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=_dev)


def _pairs(r, L, reach):
    """All ordered pairs (i, j), i != j, nearer than `reach` in the periodic box, sorted by i."""
    n = len(r)
    nc = torch.clamp(torch.floor(L / reach), min=1).to(torch.int64)
    out = []
    if int(nc.min()) < 3 or n < 2000:
        step = max(1, 40_000_000 // n)
        for s in range(0, n, step):
            d = r[None, :, :] - r[s:s + step, None, :]
            d -= L * torch.round(d / L)
            hit = (d * d).sum(-1) <= reach * reach
            i, j = torch.nonzero(hit, as_tuple=True)
            i = i + s
            keep = i != j
            out.append((i[keep], j[keep]))
    else:
        c = torch.clamp((r / L * nc).to(torch.int64), min=0)
        c = torch.minimum(c, nc - 1)
        key = (c[:, 2] * nc[1] + c[:, 1]) * nc[0] + c[:, 0]
        order = torch.argsort(key, stable=True)
        ncell = int(nc.prod())
        count = torch.bincount(key, minlength=ncell)
        most = int(count.max())
        first = torch.cumsum(count, 0) - count
        table = torch.full((ncell, most), -1, dtype=torch.int64, device=_dev)
        rank = torch.arange(n, device=_dev) - first[key[order]]
        table[key[order], rank] = order
        g = torch.arange(-1, 2, device=_dev)
        off = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
        step = max(1, 30_000_000 // (27 * most))
        for s in range(0, n, step):
            q = torch.remainder(c[s:s + step, None, :] + off[None], nc)
            cand = table[(q[..., 2] * nc[1] + q[..., 1]) * nc[0] + q[..., 0]].reshape(len(q), -1)
            i = torch.arange(s, s + len(q), device=_dev)[:, None].expand_as(cand)
            keep = (cand >= 0) & (cand != i)
            i, j = i[keep], cand[keep]
            d = r[j] - r[i]
            d -= L * torch.round(d / L)
            near = (d * d).sum(-1) <= reach * reach
            out.append((i[near], j[near]))
    return torch.cat([o[0] for o in out]), torch.cat([o[1] for o in out])


class _Spline:
    """The C2 piecewise cubic through y at k h: knot slopes from the tridiagonal system z[k-1] + 4 z[k] + z[k+1] =
    3 (y[k+1] - y[k-1]) / h, natural at the ends (they lie outside the range that is read)."""

    def __init__(self, y, h):
        n = len(y)
        d = np.empty(n)
        d[0], d[-1] = 3.0 * (y[1] - y[0]) / h, 3.0 * (y[-1] - y[-2]) / h
        d[1:-1] = 3.0 * (y[2:] - y[:-2]) / h
        b = [2.0] + [4.0] * (n - 2) + [2.0]
        z = d.tolist()
        for k in range(1, n):
            w = 1.0 / b[k - 1]
            b[k] -= w
            z[k] -= w * z[k - 1]
        z[-1] /= b[-1]
        for k in range(n - 2, -1, -1):
            z[k] = (z[k] - z[k + 1]) / b[k]
        z = np.array(z)
        m = (y[1:] - y[:-1]) / h
        # y + x (z + x (c + x e)) on each interval
        self.c = _t(np.stack([y[:-1], z[:-1], (3.0 * m - 2.0 * z[:-1] - z[1:]) / h,
                              (z[:-1] + z[1:] - 2.0 * m) / (h * h)], 1))
        self.h = h

    def __call__(self, x):
        k = torch.clamp((x / self.h).to(torch.int64), max=len(self.c) - 1)
        u = x - k.to(torch.float64) * self.h
        c = self.c[k]
        f = c[:, 0] + u * (c[:, 1] + u * (c[:, 2] + u * c[:, 3]))
        return f, c[:, 1] + u * (2.0 * c[:, 2] + 3.0 * u * c[:, 3])


class _Exact:
    """Forces, energies and virials of one system (or several side by side: L is per atom then)."""

    def __init__(self, system, kind):
        self.system, self.rc = system, SYSTEMS[system]["rc"]
        self.kind = _t(kind.astype(np.int64), torch.int64)
        if system in ("copper", "nial"):
            tabs = _tables_of(system)
            self.tab = {k: (_Spline(t["R"], t["dr"]), _Spline(t["V"], t["dr"]), _Spline(t["F"], t["drh"]))
                        for k, t in tabs.items()}

    def _chunks(self, r, L, i, j):
        step = 20_000_000
        for s in range(0, len(i), step):
            a, b = i[s:s + step], j[s:s + step]
            d = r[b] - r[a]
            box = L[a] if L.dim() == 2 else L
            d -= box * torch.round(d / box)
            r2 = (d * d).sum(-1)
            near = r2 <= self.rc * self.rc
            yield a[near], b[near], d[near], r2[near]

    def _classes(self, a, b):
        if self.system != "nial":
            yield (0, 0), slice(None)
            return
        s = self.kind[a] + self.kind[b]
        for k, key in ((0, (0, 0)), (1, (0, 1)), (2, (1, 1))):
            yield key, torch.nonzero(s == k, as_tuple=True)[0]

    def __call__(self, r, L, i, j, sample=False):
        n = len(r)
        f = torch.zeros_like(r)
        ep = torch.zeros(n, dtype=torch.float64, device=_dev)
        em = torch.zeros_like(ep)
        V = torch.zeros((n, 9), dtype=torch.float64, device=_dev)
        eam = self.system in ("copper", "nial")
        if eam:
            rho = torch.zeros_like(ep)
            for a, b, d, r2 in self._chunks(r, L, i, j):
                x = torch.sqrt(r2)
                for key, w in self._classes(a, b):
                    rho.index_add_(0, a[w], self.tab[key][0](x[w])[0])
            dF = {key: self.tab[key][2](rho) for key in self.tab}
            em = dF[0, 0][0]
            if self.system == "nial":
                # every table has the same F
                em = torch.where(self.kind == 0, dF[0, 0][0], dF[1, 1][0])
        for a, b, d, r2 in self._chunks(r, L, i, j):
            g = torch.empty_like(r2)
            e = torch.empty_like(r2)
            for key, w in self._classes(a, b):
                q = r2[w]
                if eam:
                    x = torch.sqrt(q)
                    v, dv = self.tab[key][1](x)
                    dr = self.tab[key][0](x)[1]
                    g[w] = ((dF[key][1][a[w]] + dF[key][1][b[w]]) * dr + (dv * x - v) / q) / x
                    e[w] = 0.5 * v / x
                else:
                    s6 = (SIGMA * SIGMA / q) ** 3
                    g[w] = -24.0 * EPS * s6 * (2.0 * s6 - 1.0) / q
                    e[w] = 2.0 * EPS * s6 * (s6 - 1.0)
            f.index_add_(0, a, g[:, None] * d)
            if sample:
                ep.index_add_(0, a, e)
                V.index_add_(0, a, (0.5 * g[:, None, None] * d[:, :, None] * d[:, None, :]).reshape(-1, 9))
        return (f, ep, em, V) if sample else f


def _philox(c, k):
    """Philox4x32-10 of Salmon et al. (SC'11): counters (4, n), key (2)."""
    c = [x.astype(np.uint64) for x in c]
    k = [int(k[0]), int(k[1])]
    low = np.uint64(0xFFFFFFFF)
    for rnd in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k[0]), p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k[1]),
             p0 & low]
        k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
    return c


def _langevin(n, call, v, m, p):
    """The thermostat's force at its `call`-th application: random and friction part."""
    atom = np.arange(n)
    b = _philox([atom, np.full(n, call), np.zeros(n, np.int64), np.zeros(n, np.int64)],
                (NVT["seed"] & 0xFFFFFFFF, NVT["seed"] >> 32))
    u = [(x.astype(np.float64) + 0.5) * 2.0 ** -32 for x in b]
    ra, rb = np.sqrt(-2.0 * np.log(u[0])), np.sqrt(-2.0 * np.log(u[2]))
    z = np.stack([ra * np.cos(2 * np.pi * u[1]), ra * np.sin(2 * np.pi * u[1]), rb * np.cos(2 * np.pi * u[3])], 1)
    sigma = math.sqrt(2.0 * NVT["beta"] * KB * p["T"] / p["dt"])
    return _t(z) * sigma * torch.sqrt(m) - v * NVT["beta"] * m


def _follow(system, r, v, m, kind, L, steps, nvt=False, parts=None):
    """`steps` velocity-Verlet steps from (r, v), positions wrapped into the box where the list is rebuilt: an atom
    further than half the skin from where it was at the last rebuild. `parts`: the systems lie side by side, each
    (first, last, box), with rebuilds of its own."""
    p = SYSTEMS[system]
    dt, skin = p["dt"], p["skin"]
    ex = _Exact(system, kind)
    r, v, m = _t(r), _t(v), _t(m)[:, None]
    parts = parts or [(0, len(r), L)]
    box = torch.empty_like(r)
    for a, b, e in parts:
        box[a:b] = _t(e)
    one = _t(L) if len(parts) == 1 else box
    found, near = [None] * len(parts), [None, None]

    def rebuild(which):
        for k in which:
            a, b, e = parts[k]
            i, j = _pairs(torch.remainder(r[a:b], _t(e)), _t(e), p["rc"] + skin)
            found[k] = (i + a, j + a)
        near[:] = [torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])]

    n = len(r)
    label = torch.empty(n, dtype=torch.int64, device=_dev)
    for k, (a, b, _) in enumerate(parts):
        label[a:b] = k
    r0 = r.clone()
    rebuild(range(len(parts)))
    call = 0

    def forces():
        nonlocal call
        f = ex(r, one, *near)
        if nvt:
            f = f + _langevin(n, call, v, m, p)
            call += 1
        return f

    f = forces()
    for _ in range(steps):
        v = v + f * (0.5 * dt) / m
        r = r + v * dt
        f = forces()
        v = v + f * (0.5 * dt) / m
        d = r - r0
        d -= box * torch.round(d / box)
        far = ((d * d).sum(-1) > 0.25 * skin * skin).to(torch.int64)
        due = torch.zeros(len(parts), dtype=torch.int64, device=_dev).index_add_(0, label, far) > 0
        if bool(due.any()):
            mask = due[label][:, None]
            wrapped = torch.where(r < 0, r + box, torch.where(r > box, r - box, r))
            r = torch.where(mask, wrapped, r)
            r0 = torch.where(mask, r, r0)
            rebuild([k for k, x in enumerate(due.tolist()) if x])
    return r, v, f


def exact(case, seed):
    if case["kind"] == "lists":
        return None
    if case["kind"] == "serve":
        reqs = [(q, _inputs(*q)) for q in _served(case, seed)]
        done = {}
        for system in ("argon", "copper"):
            mine = [k for k, (q, _) in enumerate(reqs) if q[0] == system]
            if not mine:
                continue
            at, parts = 0, []
            for k in mine:
                n = len(reqs[k][1][0])
                parts.append((at, at + n, reqs[k][1][4]))
                at += n
            r, v, m, kind = (np.concatenate([reqs[k][1][q] for k in mine]) for q in range(4))
            out = _follow(system, r, v, m, kind, parts[0][2], case["steps"], parts=parts)
            for k, (a, b, _) in zip(mine, parts):
                done[k] = [x[a:b] for x in out]
        return {k: torch.cat([done[q][w] for q in range(len(reqs))]) for w, k in enumerate(("r", "v", "f"))}
    r, v, m, kind, L = _inputs(case["system"], case["nx"], case["ny"], case["nz"], seed)
    if case["kind"] == "run":
        out = _follow(case["system"], r, v, m, kind, L, case["steps"], case["nvt"])
        return dict(zip(("r", "v", "f"), out))
    x, mt = _t(r), _t(m)[:, None]
    p = SYSTEMS[case["system"]]
    _, ep, em, V = _Exact(case["system"], kind)(x, _t(L), *_pairs(x, _t(L), p["rc"] + p["skin"]), sample=True)
    vcom = (mt * _t(v)).sum(0) / mt.sum()
    ke = 0.5 * (mt * (_t(v) - vcom) ** 2).sum()
    totals = {"Ep": ep.sum(), "Em": em.sum(), "KE": ke, "Etot": ep.sum() + em.sum() + ke,
              "virial": (V[:, 0] + V[:, 4] + V[:, 8]).sum(), "vcom": vcom}
    return {"Ep": ep, "Em": em if case["system"] != "argon" else torch.zeros_like(ep), "V": V, "totals": totals}

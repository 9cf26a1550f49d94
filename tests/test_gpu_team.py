"""Runs by a grid's team (one kernel for all the steps) against the loop that
launches every pass, at the edges of the sizes, blocks and buffers.

The passes' arithmetic and the order of their sums are the same, so positions,
velocities and forces must be the same bits in both precisions."""
from __future__ import annotations

import numpy as np
import pytest

import mdcraft_gb300 as mdg
from mdcraft_gb300 import workloads as W
from tests import gpu_helpers as H

pytestmark = pytest.mark.gpu

LANGEVIN = dict(beta=2.0, temperature=300.0, time_step=0.002, heat_x=1, heat_y=1, heat_z=1, Ux=0.05, seed=77)


class _Run:
    def __init__(self, kind, n, precision, per=(1, 1, 1), rns=None, thermo=None, T=None, tag0=0, ctx=None):
        ncell = max(4, int(np.ceil((max(n, 1) / 4.0) ** (1.0 / 3.0))))
        make = W.lj_argon_fcc if kind == "lj" else W.eam_cu_fcc
        atoms, box, _, p = make(ncell=ncell, jitter=0.01, **({} if T is None else {"T": T}))
        atoms = atoms[:n].copy()
        if rns is not None:
            atoms["rns"] = rns(atoms["rcut"])
        if tag0:
            atoms["tag"][::tag0] = 0
        dom = mdg.Domain(*box)
        for k in range(3):
            if per[k]:
                dom.set_periodic(k, True)
        self.sys = mdg.System(ctx or H.ctx(), dom, atoms)
        self.list = mdg.VerletList(self.sys)
        self.list.update(-1.0)
        if kind == "lj":
            pot = mdg.LJsCut(p["a"], p["s"], p["rcut"])
        else:
            t = p["tables"]
            pot = mdg.EAM(t["rcut"], t["Femb"], t["Rho"], t["Vpar"], t["Nr1"], t["dr"], t["Nrh1"], t["drh"])
        self.sol = mdg.Single(pot, periodic=True, precision=precision)
        if thermo:
            self.th = mdg.Compound(*[mdg.Langevin(**t) for t in thermo])
            self.sol.set_thermostat(self.th)
        self.keep = (dom, pot, ctx)
        self.sol.prepare(self.sys)
        self.sol.stages(self.sys)
        self.verlet, self.dt, self.atoms = mdg.Verlet(self.sol), p["dt"], atoms

    def steps(self, n, stagewise):
        if stagewise:
            H.ctx().set_timing(True)  # timed runs launch every pass
        try:
            self.verlet.run(self.sys, self.dt, n)
        finally:
            H.ctx().set_timing(False)

    def state(self):
        a = self.sys.download()
        return a, self.list.rebuilds(), self.sys.thermo_calls()


def _check(precision, batches, *args, **kw):
    out = []
    for stagewise in (False, True):
        r = _Run(*args, precision=precision, **kw)
        for n in batches:
            r.steps(n, stagewise)
        out.append(r.state())
        r.sys.close()
    (a, ra, ca), (b, rb, cb) = out
    assert ca == cb
    assert ra == rb
    for f in ("r", "v", "f"):
        assert np.array_equal(a[f], b[f]), f
    return ra


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("kind", ["lj", "eam"])
@pytest.mark.parametrize("n", [1, 2, 9, 95, 97, 607, 609, 1217])
def test_small_open_clusters(kind, n, precision):
    """From one block of one atom to a few hundred blocks' worth of nothing."""
    _check(precision, [7, 8], kind, n, per=(0, 0, 0))


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("kind", ["lj", "eam"])
@pytest.mark.parametrize("batches", [[1], [2], [1, 1, 1], [3, 1, 20]])
def test_step_counts(kind, batches, precision):
    """The positions end in their own buffers whatever the number of steps."""
    _check(precision, batches, kind, 2048)


@pytest.mark.parametrize("kind,n", [(k, n) for k in ("lj", "eam") for n in (40736, 40737, 116735, 116736)])
def test_rule_edges_mixed(kind, n):
    _check("mixed", [6], kind, n)


@pytest.mark.parametrize("kind,n", [("lj", 1999), ("lj", 2000), ("lj", 23999), ("lj", 24000), ("eam", 1999), ("eam", 2000),
                                    ("eam", 12499), ("eam", 12500)])
def test_rule_edges_fp64(kind, n):
    _check("fp64", [6], kind, n)


@pytest.mark.parametrize("kind", ["lj", "eam"])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_thermostat_and_tag0(kind, precision):
    terms = [LANGEVIN, dict(LANGEVIN, seed=5, heat_y=0, xmin=0.3, xmax=1.9)]
    _check(precision, [9, 10], kind, 2916, thermo=terms, tag0=7)


@pytest.mark.parametrize("kind", ["lj", "eam"])
def test_rebuilds(kind):
    """Hot atoms and a thin skin: a rebuild every step or two."""
    n = _check("mixed", [40, 21], kind, 4000, T=3000.0, rns=lambda rc: rc + 0.004)
    assert n >= 20


def test_votes_of_many_barriers():
    """Enough barriers at which most blocks vote that the counts of votes pass
    their field's top bit (2^15) several times."""
    n = _check("mixed", [1500], "lj", 2048, T=1500.0, rns=lambda rc: rc + 1e-5)
    assert n >= 1000


@pytest.mark.parametrize("kind,precision", [("lj", "mixed"), ("lj", "fp64"), ("eam", "mixed")])
def test_list_outgrown_during_a_run(kind, precision):
    """Atoms that fall together: a rebuild needs more room than there is, the
    kernel ends early and the rest of the steps resume."""
    out = []
    for stagewise in (False, True):
        r = _Run(kind, 1372, precision, per=(0, 0, 0))
        r0 = r.atoms["r"]
        c = r0.mean(axis=0)
        r.sys.set_positions(c + 3.0 * (r0 - c) * 0.45)
        r.list.update(-1.0)
        r.sys.set_velocities(-(r0 - c) * 0.5 / (60 * r.dt))
        first = r.list.total()
        r.steps(60, stagewise)
        out.append((r.state(), first, r.list.total()))
        r.sys.close()
    ((a, ra, _), t0, t1), ((b, rb, _), _, t2) = out
    assert t1 == t2 > t0
    assert ra == rb
    assert np.array_equal(a["r"], b["r"]) and np.array_equal(a["v"], b["v"])


@pytest.mark.parametrize("steps", [255, 256, 257, 513])
@pytest.mark.parametrize("pinned", [False, True])
def test_launches_of_256_steps(steps, pinned):
    a, b = _Run("lj", 864, "mixed"), _Run("lj", 864, "mixed")
    a.steps(steps, True)
    ref = a.sys.download()
    if pinned:
        pos, vel = _pinned(b.atoms["r"]), _pinned(b.atoms["v"])
        b.verlet.run_host(b.sys, b.dt, steps, pos.numpy(), vel.numpy())
        assert np.array_equal(pos.numpy(), ref["r"]) and np.array_equal(vel.numpy(), ref["v"])
    else:
        b.steps(steps, False)
    got = b.sys.download()
    for f in ("r", "v", "f"):
        assert np.array_equal(got[f], ref[f]), f
    a.sys.close()
    b.sys.close()


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_threads_share_the_device(precision):
    """Runs of four threads, each on its own system and context: whichever of
    them runs alone, the bits are those of launched passes."""
    import threading
    ref = _Run("lj", 2048, precision)
    ref.steps(600, True)
    want = ref.sys.download()
    runs = [_Run("lj", 2048, precision, ctx=mdg.Context(0)) for _ in range(4)]
    threads = [threading.Thread(target=r.verlet.run, args=(r.sys, r.dt, 600)) for r in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for r in runs:
        got = r.sys.download()
        for f in ("r", "v", "f"):
            assert np.array_equal(got[f], want[f]), f
        r.sys.close()
    ref.sys.close()


def _pinned(x):
    import torch
    t = torch.empty(np.shape(x), dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = x
    return t


@pytest.mark.parametrize("kind", ["lj", "eam"])
@pytest.mark.parametrize("n,steps", [(500, 30), (16385, 30), (27999, 1), (28000, 1), (28000, 2), (44000, 2), (44001, 2)])
@pytest.mark.parametrize("force", [False, True])
def test_host_arrays(kind, n, steps, force):
    """Page-locked host arrays, which the kernel reads and writes itself (and
    28,000 atoms' one-step calls the overlapped step), against a run and its
    downloads."""
    a, b = _Run(kind, n, "mixed", tag0=11), _Run(kind, n, "mixed", tag0=11)
    a.steps(steps, True)
    ref = a.sys.download()
    pos, vel, frc = _pinned(b.atoms["r"]), _pinned(b.atoms["v"]), _pinned(np.zeros_like(b.atoms["r"]))
    b.verlet.run_host(b.sys, b.dt, steps, pos.numpy(), vel.numpy(), frc.numpy() if force else None)
    assert np.array_equal(pos.numpy(), ref["r"])
    assert np.array_equal(vel.numpy(), ref["v"])
    assert np.array_equal(frc.numpy() if force else b.sys.forces(), ref["f"])
    a.sys.close()
    b.sys.close()


@pytest.mark.parametrize("kind", ["lj", "eam"])
def test_precisions_in_turn(kind):
    """Mixed and FP64 runs in turn on one system."""
    out = []
    for stagewise in (False, True):
        r = _Run(kind, 2048, "mixed")
        for prec in ("mixed", "fp64", "mixed", "fp64", "mixed"):
            r.sol.set_precision(prec)
            r.steps(5, stagewise)
        out.append(r.state()[0])
        r.sys.close()
    for f in ("r", "v", "f"):
        assert np.array_equal(out[0][f], out[1][f]), f

"""The graph loop's passes that start the next step (the LJ pass, which moves
atoms between two sets of arrays, and the thermostat's) against the loop that
launches every pass: the same bits, after any number of steps and through
rebuilds, ends of runs and lists that outgrow their room."""
from __future__ import annotations

import numpy as np
import pytest

import mdcraft_gb300 as mdg
from mdcraft_gb300 import workloads as W
from tests import gpu_helpers as H

pytestmark = pytest.mark.gpu

LANGEVIN = dict(beta=2.0, temperature=300.0, time_step=0.002, heat_x=1, heat_y=1, heat_z=1, Ux=0.05, seed=77)


def _run(kind, n, batches, stagewise, thermo=None, T=100.0, skin=None, tag0=13, squeeze=0.0):
    ncell = int(np.ceil((n / 4.0) ** (1.0 / 3.0)))
    if kind == "eam":
        atoms, box, _, p = W.eam_cu_fcc(ncell=ncell, jitter=0.01, T=T)
        t = p["tables"]
        pots = [mdg.EAM(t["rcut"], t["Femb"], t["Rho"], t["Vpar"], t["Nr1"], t["dr"], t["Nrh1"], t["drh"])]
        sol = mdg.Single(pots[0], periodic=True, precision="mixed")
    else:
        atoms, box, _, p = W.lj_argon_fcc(ncell=ncell, jitter=0.01, T=T)
        pots = [mdg.LJsCut(p["a"] * (1.0 + 0.01 * k), p["s"], p["rcut"]) for k in range(3)]
        if kind == "lj":
            sol = mdg.Single(pots[0], periodic=True, precision="mixed")
        else:
            atoms["kind"] = np.arange(len(atoms)) % 2
            sol = mdg.Multi(2, periodic=True, precision="mixed")
            for k, (i, j) in enumerate(((0, 0), (0, 1), (1, 1))):
                sol.add_potential(i, j, pots[k])
    atoms = atoms[:n].copy()
    atoms["tag"][::tag0] = 0
    if skin is not None:
        atoms["rns"] = atoms["rcut"] + skin
    dom = mdg.Domain(*box)
    for k in range(3):
        dom.set_periodic(k, True)
    ctx = H.ctx()
    sys = mdg.System(ctx, dom, atoms)
    nl = mdg.VerletList(sys)
    if squeeze:
        c = atoms["r"].mean(axis=0)
        sys.set_velocities(-(atoms["r"] - c) * squeeze / (sum(batches) * p["dt"]))
    nl.update(-1.0)
    if thermo:
        th = mdg.Compound(*[mdg.Langevin(**t) for t in thermo])
        sol.set_thermostat(th)
    sol.prepare(sys)
    sol.stages(sys)
    v = mdg.Verlet(sol)
    if stagewise:
        ctx.set_timing(True)  # timed runs launch every pass
    try:
        for steps in batches:
            v.run(sys, p["dt"], steps)
    finally:
        ctx.set_timing(False)
    out = sys.download(), nl.rebuilds(), sys.thermo_calls(), nl.total()
    sys.close()
    return out


def _same(*args, **kw):
    (a, ra, ca, ta), (b, rb, cb, tb) = (_run(*args, stagewise=s, **kw) for s in (False, True))
    assert (ra, ca, ta) == (rb, cb, tb)
    for f in ("r", "v", "f"):
        assert np.array_equal(a[f], b[f]), f
    return ra


@pytest.mark.parametrize("kind,n", [("lj", 116737), ("lj2", 24001)])
@pytest.mark.parametrize("batches", [[1], [2], [3, 1, 2, 4]])
def test_lj_step_counts(kind, n, batches):
    _same(kind, n, batches)


@pytest.mark.parametrize("kind,n", [("lj", 116737), ("lj2", 30011)])
def test_lj_rebuilds(kind, n):
    assert _same(kind, n, [9, 16], T=3000.0, skin=0.01) >= 8


def test_lj_list_outgrown():
    _same("lj", 116737, [40], squeeze=0.25, tag0=1 << 30)


@pytest.mark.parametrize("kind,n", [("eam", 116737), ("lj", 116737), ("lj2", 3001)])
@pytest.mark.parametrize("batches", [[1], [2, 3], [20]])
def test_thermostat_steps(kind, n, batches):
    _same(kind, n, batches, thermo=[LANGEVIN, dict(LANGEVIN, seed=5, heat_y=0, xmin=0.3, xmax=1.9)], T=1500.0,
          skin=0.02)

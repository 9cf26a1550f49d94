"""Runs of small systems on grids of many, mostly empty bins: a crystal in a
large box with one atom in each of two far corners. Below the rule's line a
grid's team takes the run, above it the launched loop, with the same bits as
the loop that launches every pass."""
from __future__ import annotations

import numpy as np
import pytest

import mdcraft_gb300 as mdg
from mdcraft_gb300 import workloads as W
from tests import gpu_helpers as H

pytestmark = pytest.mark.gpu


class _Cluster:
    def __init__(self, ncell, cells, precision):
        atoms, box, _, p = W.lj_argon_fcc(ncell=ncell, jitter=0.01)
        rns = p["rcut"] + 0.01
        L = cells * rns * 1.0001
        atoms["rns"] = rns
        atoms["r"] += (L - box[1]) / 2
        atoms["r"][0], atoms["r"][-1] = 0.01, L - 0.5 * rns
        atoms["tag"][[0, -1]] = 0
        d = mdg.Domain(0, L, 0, L, 0, L)
        for k in range(3):
            d.set_periodic(k, True)
        self.sys = mdg.System(H.ctx(), d, atoms)
        self.list = mdg.VerletList(self.sys)
        self.list.update(-1.0)
        self.sol = mdg.Single(mdg.LJsCut(p["a"], p["s"], p["rcut"]), periodic=True, precision=precision)
        self.sol.prepare(self.sys)
        self.sol.stages(self.sys)
        self.verlet, self.dt, self.keep = mdg.Verlet(self.sol), p["dt"], d

    def run(self, steps, stagewise):
        H.ctx().set_timing(stagewise)  # timed runs launch every pass
        before = H.ctx().launches()
        self.verlet.run(self.sys, self.dt, steps)
        H.ctx().set_timing(False)
        a = self.sys.download()
        return [a[f].copy() for f in ("r", "v", "f")], self.list.rebuilds(), H.ctx().launches() - before


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("ncell,cells,team", [(10, 40, True), (10, 44, False), (18, 44, False), (19, 32, None), (19, 36, False)])
def test_bins(ncell, cells, team, precision):
    out = []
    for stagewise in (False, True):
        c = _Cluster(ncell, cells, precision)
        out.append(c.run(30, stagewise))
        c.sys.close()
    (a, ra, launches), (b, rb, _) = out
    assert ra == rb and ra > 1
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    if team is None:
        team = precision == "mixed"  # 27,436 atoms: above the FP64 rule
    assert (launches < 10) == team

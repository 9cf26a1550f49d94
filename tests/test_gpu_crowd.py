"""Systems run by several threads at once, few enough and too many for a GPU of
their own (run_crowded): the same bits as a system run alone, over runs that go
back and forth between the two."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import mdcraft_gb300 as mdg
from mdcraft_gb300 import workloads as W
from tests import gpu_helpers as H
from tests.test_gpu_team import _Run

pytestmark = pytest.mark.gpu


class _Alloy(_Run):
    def __init__(self, n, ctx):
        atoms, box, _, p = W.eam_nial_b2(ncell=20)
        atoms = atoms[:n].copy()
        dom = mdg.Domain(*box)
        for k in range(3):
            dom.set_periodic(k, True)
        self.sys = mdg.System(ctx, dom, atoms)
        self.list = mdg.VerletList(self.sys)
        self.list.update(-1.0)
        self.sol = mdg.Multi(2, periodic=True, precision="mixed")
        pots = []
        for (i, j), t in p["tables"].items():
            pots.append(mdg.EAM(t["rcut"], t["Femb"], t["Rho"], t["Vpar"], t["Nr1"], t["dr"], t["Nrh1"], t["drh"]))
            self.sol.add_potential(i, j, pots[-1])
        self.keep = (dom, pots, ctx)
        self.sol.prepare(self.sys)
        self.sol.stages(self.sys)
        self.verlet, self.dt, self.atoms = mdg.Verlet(self.sol), p["dt"], atoms


def _make(kind, n):
    ctx = mdg.Context(0)
    if kind == "nial":
        return _Alloy(n, ctx)
    return _Run(kind, n, precision="mixed", T=900.0, rns=lambda rc: rc + 0.01, ctx=ctx)


@pytest.mark.parametrize("kind,n", [("lj", 13500), ("eam", 13500), ("nial", 15000)])
def test_crowds_have_the_bits_of_one(kind, n):
    H.ctx()
    alone = _make(kind, n)
    for _ in range(4):
        alone.verlet.run(alone.sys, alone.dt, 30)
    want, rebuilds, _ = alone.state()
    alone.sys.close()
    runs = [_make(kind, n) for _ in range(8)]
    # one, eight, three, eight at a time: 70,000 atoms is a crowd
    for many in (1, 8, 3, 8):
        for k in range(0, 8, many):
            start = threading.Barrier(len(runs[k:k + many]))

            def work(r):
                start.wait()
                r.verlet.run(r.sys, r.dt, 30)

            threads = [threading.Thread(target=work, args=(r,)) for r in runs[k:k + many]]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
    for r in runs:
        got, rb, _ = r.state()
        assert rb == rebuilds
        for f in ("r", "v", "f"):
            assert np.array_equal(got[f], want[f]), f
        r.sys.close()

"""Served requests by teams of blocks (few requests outstanding) against one
block of the persistent kernel each (a block size asked for): the same bits,
for any number of requests and sizes, across the change from one to the other
and for a request whose list outgrows its room."""
from __future__ import annotations

import numpy as np
import pytest

import mdcraft_gb300 as mdg
from mdcraft_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _requests(count, n_max, seed):
    rng = np.random.default_rng(seed)
    out = []
    for k in range(count):
        n = int(np.exp(rng.uniform(np.log(8), np.log(n_max))))
        kind = "lj" if k % 3 else "eam"
        ncell = max(5, int(np.ceil((n / 4.0) ** (1.0 / 3.0))))
        make = W.lj_argon_fcc if kind == "lj" else W.eam_cu_fcc
        atoms, box, _, p = make(ncell=ncell, jitter=0.01, T=600.0, seed=k + 1)
        atoms = atoms[:n].copy()
        if k % 5 == 0:
            atoms["rns"] = atoms["rcut"] + 0.01  # many rebuilds
        out.append((kind, atoms, box, p))
    return out


def _solvers():
    _, _, _, p = W.lj_argon_fcc(ncell=5)
    _, _, _, q = W.eam_cu_fcc(ncell=5)
    t = q["tables"]
    pots = dict(lj=mdg.LJsCut(p["a"], p["s"], p["rcut"]),
                eam=mdg.EAM(t["rcut"], t["Femb"], t["Rho"], t["Vpar"], t["Nr1"], t["dr"], t["Nrh1"], t["drh"]))
    return pots, {k: mdg.Single(v, periodic=True, precision="mixed") for k, v in pots.items()}


def _serve(reqs, block_threads, steps, waves=1):
    pots, solvers = _solvers()
    server = mdg.Server(slots=64, max_atoms=16384, block_threads=block_threads)
    got = []
    for w in range(waves):
        part = reqs[w::waves]
        ids = []
        for kind, atoms, box, p in part:
            dom = mdg.Domain(*box)
            for k in range(3):
                dom.set_periodic(k, True)
            ids.append(server.submit(solvers[kind], dom, atoms, p["dt"], steps))
        for i in ids:
            server.wait(i, 60.0)
            at, info = server.result(i)
            assert info["status"] == 0
            got.append((at, info["rebuilds"]))
    server.close()
    return got


@pytest.mark.parametrize("count,n_max", [(1, 5000), (2, 9), (7, 4000), (48, 3000), (76, 600), (77, 600), (200, 600)])
def test_teams_equal_single_blocks(count, n_max):
    reqs = _requests(count, n_max, seed=count)
    for (a, ra), (b, rb) in zip(_serve(reqs, 0, 25), _serve(reqs, 512, 25)):
        assert ra == rb
        assert a.tobytes() == b.tobytes()


def test_waves_reuse_slots():
    """The same slots, scratch and streams by one wave of requests after another."""
    reqs = _requests(30, 2000, seed=5)
    for (a, ra), (b, rb) in zip(_serve(reqs, 0, 7, waves=6), _serve(reqs, 640, 7, waves=6)):
        assert ra == rb
        assert a.tobytes() == b.tobytes()


def test_list_outgrown():
    """Atoms that fall together outgrow the list sized at admission: the run is
    void and repeated on the checked path."""
    atoms, box, _, p = W.lj_argon_fcc(ncell=8, jitter=0.01)
    c = atoms["r"].mean(axis=0)
    L = box[1] - box[0]
    box = tuple(v + (L if k % 2 else -L) for k, v in enumerate(box))
    atoms["v"] = -(atoms["r"] - c) * 0.25 / (40 * p["dt"])
    reqs = [("lj", atoms, box, p)]
    (a, ra), = _serve(reqs, 0, 40)
    (b, rb), = _serve(reqs, 512, 40)
    assert ra == rb
    assert a.tobytes() == b.tobytes()


def test_thermostat_and_tabulated_pair_take_the_graph():
    """Requests that the fused loops do not carry give the plain API's bits."""
    from tests import gpu_helpers as H
    atoms, box, _, p = W.lj_argon_fcc(ncell=5, jitter=0.01)
    dom = mdg.Domain(*box)
    for k in range(3):
        dom.set_periodic(k, True)
    r = np.linspace(0.0, 1.1 * p["rcut"], 2001)
    table = r * np.exp(-r / 0.2)
    pots = [mdg.LJsCut(p["a"], p["s"], p["rcut"]), mdg.Pair(p["rcut"], table, len(r) - 1, r[1])]
    for pot, thermo in ((pots[0], True), (pots[1], False)):
        sol = mdg.Single(pot, periodic=True, precision="mixed")
        if thermo:
            th = mdg.Langevin(2.0, 300.0, p["dt"], seed=9)
            sol.set_thermostat(th)
        server = mdg.Server(slots=4, max_atoms=1024)
        rid = server.submit(sol, dom, atoms, p["dt"], 20)
        server.wait(rid, 60.0)
        got, info = server.result(rid)
        assert info["status"] == 0
        server.close()
        s = mdg.System(H.ctx(), dom, atoms)
        mdg.VerletList(s).update(-1.0)
        sol.prepare(s)
        sol.stages(s)
        # the request's initial forces count as a thermostat call, as here
        mdg.Verlet(sol).run(s, p["dt"], 20)
        want = s.download()
        for f in ("r", "v"):
            assert np.array_equal(got[f], want[f]), f
        s.close()

"""Lists of grids with an axis of two cells ("flat") and of grids short of a
periodic box ("short"), on both sides of the line between a warp and a thread
per atom (atoms_by_threads, block_by_threads): neighbour sets as the oracle's,
requests with the bits of the launched loop."""
from __future__ import annotations

import numpy as np
import pytest

import mdcraft_gb300 as mdg
from mdcraft_gb300 import workloads as W
from oracle import mdref as R
from tests import gpu_helpers as H
from tests.test_gpu_rebuild import _gas, _same_lists
from tests.test_gpu_serving_team import _solvers

pytestmark = pytest.mark.gpu


def _flat(n, per_cell):
    """A gas in a box of 2 x m x m cells."""
    m = max(3, int(round((n / per_cell / 2) ** 0.5)))
    L = np.array([2, m, m]) + 0.01
    a, _ = _gas(n, 1.0, 1.0, seed=n)
    a["r"] = np.random.default_rng(n).uniform(0.0, 1.0, (n, 3)) * L
    return a, (0.0, L[0], 0.0, L[1], 0.0, L[2])


def _short(n, per_cell):
    """A gas in the middle of a larger periodic box."""
    m = max(3, int(round((n / per_cell) ** (1 / 3))))
    a, _ = _gas(n, m + 0.01, 1.0, seed=n)
    a["r"] += 1.5
    L = m + 3.0
    return a, (0.0, L, 0.0, L, 0.0, L)


# lines: flat 12,000 + 950 a cell's atom, short 3,000 + 1,000
@pytest.mark.parametrize("make,per_cell,n", [(_flat, 4, 14500), (_flat, 4, 17500), (_flat, 20, 27000), (_flat, 20, 36000),
                                             (_short, 4, 6000), (_short, 4, 9000), (_short, 12, 13000), (_short, 12, 18000)])
def test_both_sides_of_the_line(make, per_cell, n):
    _same_lists(*make(n, per_cell))


@pytest.mark.parametrize("make,n", [(_flat, 17500), (_short, 9000)])
def test_uneven_rns_by_threads(make, n):
    a, box = make(n, 4)
    a["rns"] = np.random.default_rng(2).uniform(0.6, 1.0, n)
    a["rns"][0] = 1.0
    a["rcut"] = 0.9 * a["rns"]
    _same_lists(a, box)


@pytest.mark.parametrize("make,n", [(_flat, 17500), (_short, 9000)])
def test_half_list_by_threads(make, n):
    a, box = make(n, 4)
    d, do = mdg.Domain(*box), R.Domain(*box)
    for k in range(3):
        d.set_periodic(k, True)
        do.set_periodic(k, True)
    s = mdg.System(H.ctx(), d, a)
    nl = mdg.VerletList(s, half=True)
    nl.update(-1.0)
    no = R.VerletList(H.to_oracle_atoms(a), do, half=True, threads=1)
    no.update(-1.0)
    assert H.same_sets(nl.lists(), no.lists()) == 0
    s.close()


def test_clamped_atoms_by_threads():
    """A slab open in z in a periodic box it does not fill, atoms beyond it."""
    a, box = _short(9000, 4)
    z = a["r"][:, 2]
    _same_lists(a, (*box[:4], float(np.quantile(z, 0.02)), float(np.quantile(z, 0.98))), per=(1, 1, 0))


@pytest.mark.parametrize("threads", [256, 640])
@pytest.mark.parametrize("off", [-1, 0, 1])
def test_requests_in_one_block(threads, off):
    """Half the block's threads with an atom, one fewer and one more; the flat
    box has two cells on one axis."""
    n = threads // 2 + off
    atoms, box, _, p = W.lj_argon_fcc(ncell=8, jitter=0.01, T=600.0)
    lay = atoms["r"][:, 2] < 4 * 0.526
    atoms = atoms[lay][:n].copy()
    atoms["rns"] = p["rcut"] + 0.01
    dom = mdg.Domain(*box[:4], 0.0, 4 * 0.526)
    for k in range(3):
        dom.set_periodic(k, True)
    out = []
    for bt in (threads, -1):
        pots, solvers = _solvers()
        server = mdg.Server(slots=4, max_atoms=4096, block_threads=bt)
        i = server.submit(solvers["lj"], dom, atoms, p["dt"], 60)
        server.wait(i, 60.0)
        at, info = server.result(i)
        assert info["status"] == 0 and info["rebuilds"] > 3
        out.append(at)
        server.close()
    for f in ("r", "v", "f"):
        assert np.array_equal(out[0][f], out[1][f]), f


@pytest.mark.parametrize("n", [20000, 40000, 60000])
def test_team_runs_on_flat_boxes(n):
    """Both sides of the team's line, against the loop that launches every pass."""
    out = []
    for stagewise in (False, True):
        nx = int((n / 16) ** 0.5)
        atoms, box, _, p = W.lj_argon_fcc(ncell=nx, jitter=0.01, T=900.0)
        keep = atoms["r"][:, 2] < 4 * 0.526
        atoms = atoms[keep].copy()
        atoms["uid"] = np.arange(len(atoms))
        atoms["rns"] = p["rcut"] + 0.01
        dom = mdg.Domain(*box[:4], 0.0, 4 * 0.526)
        for k in range(3):
            dom.set_periodic(k, True)
        s = mdg.System(H.ctx(), dom, atoms)
        nl = mdg.VerletList(s)
        nl.update(-1.0)
        sol = mdg.Single(mdg.LJsCut(p["a"], p["s"], p["rcut"]), periodic=True, precision="mixed")
        sol.prepare(s)
        sol.stages(s)
        H.ctx().set_timing(stagewise)
        mdg.Verlet(sol).run(s, p["dt"], 15)
        H.ctx().set_timing(False)
        out.append((s.download(), nl.rebuilds()))
        s.close()
    (a, ra), (b, rb) = out
    assert ra == rb and ra > 2
    for f in ("r", "v", "f"):
        assert np.array_equal(a[f], b[f]), f

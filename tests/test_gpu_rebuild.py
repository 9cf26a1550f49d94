"""The rebuild's kernels at the edges of their rules: warps per cell (system
size), turns of eight chunks (cells of one to a hundred atoms, up to some
2,700 candidates), odd and over-32 batches, one-block and three-pass scans of
the bins, bins of many atoms in random caller order. Neighbour sets must equal
the oracle's, which are compared as whole numbers."""
from __future__ import annotations

import numpy as np
import pytest

import mdcraft_gb300 as mdg
from mdcraft_gb300 import workloads as W
from oracle import mdref as R

pytestmark = pytest.mark.gpu


def _same_lists(atoms, box, per=(1, 1, 1)):
    from tests import gpu_helpers as H
    dg, do = mdg.Domain(*box), R.Domain(*box)
    for k in range(3):
        if per[k]:
            dg.set_periodic(k, True)
            do.set_periodic(k, True)
    s = mdg.System(H.ctx(), dg, atoms)
    nl = mdg.VerletList(s)
    nl.update(-1.0)
    a = np.zeros(len(atoms), dtype=R.ATOM_DTYPE)
    a.view(np.uint8)[:] = np.ascontiguousarray(atoms).view(np.uint8)
    no = R.VerletList(a, do, threads=R.hardware_threads())
    no.update(-1.0)
    og, ig = nl.csr()
    oo, io = no.csr()
    assert np.array_equal(og, oo)
    io = np.concatenate([np.sort(io[oo[k]:oo[k + 1]]) for k in range(len(atoms))])
    assert np.array_equal(ig, io)
    assert np.array_equal(s.positions(), a["r"])
    s.close()


def _gas(n, L, rns, seed, per=(1, 1, 1)):
    rng = np.random.default_rng(seed)
    a = mdg.new_atoms(n)
    a["r"] = rng.uniform(0.0, L, (n, 3))
    a["m"] = 1.0
    a["rcut"], a["rns"] = 0.9 * rns, rns
    a["uid"] = np.arange(n)
    return a, (0.0, L, 0.0, L, 0.0, L)


@pytest.mark.parametrize("per_cell", [0.05, 0.4, 1, 7, 31, 33, 64, 100])
def test_cells_of_any_filling(per_cell):
    """4 cells per axis and about per_cell atoms in each (20 cells per axis
    where they are nearly empty, which takes the three-pass scan)."""
    cells = 4 if per_cell >= 1 else 30
    n = max(2, int(per_cell * cells ** 3))
    a, box = _gas(n, float(cells) + 0.01, 1.0, seed=int(per_cell * 100))
    _same_lists(a, box)


@pytest.mark.parametrize("n", [11999, 12000, 12001])
def test_warps_per_cell_rule(n):
    a, box = _gas(n, 9.0, 1.0, seed=n)
    _same_lists(a, box)


def test_open_axis_and_shuffled_order():
    """A slab open in z with atoms beyond the domain, in random caller order."""
    atoms, box, _, _ = W.lj_argon_fcc(ncell=7, jitter=0.05)
    rng = np.random.default_rng(5)
    atoms = atoms[rng.permutation(len(atoms))]
    box = (*box[:4], 0.4, box[5] - 0.3)
    _same_lists(atoms, box, per=(1, 1, 0))


def test_uneven_rns():
    """Atoms with list radii of their own: every pair goes to the exact test."""
    a, box = _gas(3000, 6.0, 1.0, seed=9)
    a["rns"] = np.random.default_rng(2).uniform(0.6, 1.0, len(a))
    a["rcut"] = 0.9 * a["rns"]
    _same_lists(a, box)


def test_small_boxes_warp_per_atom():
    for n, cells in ((40, 1), (300, 2), (1100, 2)):
        a, box = _gas(n, cells + 0.3, 1.0, seed=n)
        _same_lists(a, box)

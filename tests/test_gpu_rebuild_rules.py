"""The rebuild at the lines of its rules as they are: lists by a warp per atom
below 8,000 atoms and by a warp per cell from there on, there with cells of one
to a hundred atoms (batches of up to 32, shared appending, turns of 16 chunks of
candidates), radii of the atoms' own and half lists; the one-block scan up to
16,384 bins of capacity; one to four warps a cell in a grid's team.

Neighbour sets must equal the oracle's, runs the bits of the launched loop."""
from __future__ import annotations

import numpy as np
import pytest

import mdcraft_gb300 as mdg
from oracle import mdref as R
from tests import gpu_helpers as H
from tests.test_gpu_rebuild import _gas, _same_lists
from tests.test_gpu_team import _check

pytestmark = pytest.mark.gpu
FEW = 8000  # kAtomBuildMost


@pytest.mark.parametrize("n", [FEW - 1, FEW, FEW + 1])
def test_warp_per_atom_or_per_cell(n):
    a, box = _gas(n, 9.0, 1.0, seed=n)
    _same_lists(a, box)


@pytest.mark.parametrize("per_cell", [0.4, 1, 3, 7, 9, 10, 15, 17, 31, 33, 64, 100])
def test_cells_of_any_filling_by_warps(per_cell):
    cells = int(np.ceil((FEW / per_cell) ** (1.0 / 3.0)))
    n = max(FEW, int(per_cell * cells ** 3))
    a, box = _gas(n, cells + 0.01, 1.0, seed=int(per_cell * 100))
    _same_lists(a, box)


@pytest.mark.parametrize("per_cell", [7, 40])
def test_uneven_rns_by_warps(per_cell):
    cells = int(np.ceil((FEW / per_cell) ** (1.0 / 3.0)))
    a, box = _gas(per_cell * cells ** 3, cells + 0.01, 1.0, seed=per_cell)
    a["rns"] = np.random.default_rng(2).uniform(0.6, 1.0, len(a))
    a["rcut"] = 0.9 * a["rns"]
    _same_lists(a, box)


@pytest.mark.parametrize("per_cell", [7, 40])
def test_half_list_by_warps(per_cell):
    cells = int(np.ceil((FEW / per_cell) ** (1.0 / 3.0)))
    a, box = _gas(per_cell * cells ** 3, cells + 0.01, 1.0, seed=per_cell + 1)
    d, do = mdg.Domain(*box), R.Domain(*box)
    for k in range(3):
        d.set_periodic(k, True)
        do.set_periodic(k, True)
    s = mdg.System(H.ctx(), d, a)
    nl = mdg.VerletList(s, half=True)
    nl.update(-1.0)
    no = R.VerletList(H.to_oracle_atoms(a), do, half=True, threads=1)  # (it takes half lists with one thread)
    no.update(-1.0)
    assert H.same_sets(nl.lists(), no.lists()) == 0
    s.close()


@pytest.mark.parametrize("cells", [(20, 20, 20), (24, 20, 20), (24, 24, 20), (24, 24, 24)])
def test_scans_by_one_block_and_by_many(cells):
    """Capacities of 13,097, 14,897, 17,057 and 19,649 bins."""
    rng = np.random.default_rng(sum(cells))
    L = np.array(cells) + 0.01
    a, _ = _gas(FEW + 200, 1.0, 1.0, seed=1)
    a["r"] = rng.uniform(0.0, 1.0, (len(a), 3)) * L
    _same_lists(a, (0.0, L[0], 0.0, L[1], 0.0, L[2]))


@pytest.mark.parametrize("kind", ["lj", "eam"])
@pytest.mark.parametrize("n", [7999, 8000, 14593, 19457, 29185])
def test_team_parts(n, kind):
    """On 152 SMs: by atoms, then four, three, two and one warps a cell."""
    rebuilds = _check("mixed", [14], kind, n, T=3000.0, rns=lambda rc: rc + 0.004)
    assert rebuilds > 4

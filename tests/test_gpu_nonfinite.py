"""A position that is not a number, of either sign, on a list that is there
already: every force it takes part in is not a number and the flag is up."""
from __future__ import annotations

import numpy as np
import pytest

import mdcraft_gb300 as mdg
from mdcraft_gb300 import workloads as W
from tests import gpu_helpers as H

pytestmark = pytest.mark.gpu
NONFINITE = 8


@pytest.mark.parametrize("ncell", [5, 10, 15])  # 32, 16 and 4 lanes an atom
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_nan_position_is_flagged(sign, ncell):
    atoms, box, _, p = W.lj_argon_fcc(ncell=ncell, jitter=0.01)
    d = mdg.Domain(*box)
    for k in range(3):
        d.set_periodic(k, True)
    s = mdg.System(H.ctx(), d, atoms)
    nl = mdg.VerletList(s)
    nl.update(-1.0)
    lists = nl.lists()
    sol = mdg.Single(mdg.LJsCut(p["a"], p["s"], p["rcut"]), periodic=True, precision="fp64")
    sol.prepare(s)
    sol.stages(s)
    assert np.isfinite(s.forces()).all() and not s.flags() & NONFINITE
    r = s.positions()
    r[7, 1] = np.copysign(np.nan, sign)
    s.set_positions(r)
    sol.stages(s)
    hit = sorted({7, *(int(j) for j in lists[7])})
    assert sorted(np.flatnonzero(np.isnan(s.forces()[:, 1]))) == hit
    assert s.flags() & NONFINITE
    s.close()

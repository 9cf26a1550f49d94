"""Verlet.run_host on page-locked arrays that lie off an 8-byte boundary (a
record's fields, a view into a message buffer): copied, not read in place."""
from __future__ import annotations

import numpy as np
import pytest

import mdcraft_gb300 as mdg
from mdcraft_gb300 import workloads as W
from tests import gpu_helpers as H

pytestmark = pytest.mark.gpu


def _locked(a, offset):
    """A page-locked copy of `a`, `offset` bytes into its buffer."""
    import torch
    buf = torch.empty(a.nbytes + 64, dtype=torch.uint8, pin_memory=True).numpy()
    out = np.frombuffer(buf.data, dtype=np.float64, count=a.size, offset=offset).reshape(a.shape)
    out[...] = a
    assert out.ctypes.data % 8 == offset % 8
    return out


def _run(precision, steps, offsets):
    atoms, box, _, p = W.lj_argon_fcc(ncell=6, jitter=0.01)
    d = mdg.Domain(*box)
    for k in range(3):
        d.set_periodic(k, True)
    s = mdg.System(H.ctx(), d, atoms)
    mdg.VerletList(s).update(-1.0)
    sol = mdg.Single(mdg.LJsCut(p["a"], p["s"], p["rcut"]), periodic=True, precision=precision)
    sol.prepare(s)
    sol.stages(s)
    arrays = [_locked(a, o) for a, o in zip((s.positions(), s.velocities(), s.forces()), offsets)]
    mdg.Verlet(sol).run_host(s, p["dt"], steps, *arrays)
    s.close()
    return [a.copy() for a in arrays]


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("steps", [1, 5])
@pytest.mark.parametrize("offsets", [(4, 4, 4), (4, 0, 0), (0, 1, 0), (0, 0, 2), (8, 16, 24)])
def test_arrays_off_the_boundary(offsets, steps, precision):
    for a, b in zip(_run(precision, steps, offsets), _run(precision, steps, (0, 0, 0))):
        assert np.array_equal(a, b)

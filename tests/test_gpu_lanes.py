"""The mixed force passes with eight lanes per atom: block and list-length
remainders, and both sides of the rule that picks them, against the FP64 form.

Tolerance: the mixed form's own gate, 1e-5 of the forces' L2 norm (pair terms
rounded to FP32, compensated sums)."""
from __future__ import annotations

import numpy as np
import pytest

import mdcraft_gb300 as mdg
from mdcraft_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _forces(atoms, box, make, precision, per=(1, 1, 1)):
    from tests import gpu_helpers as H
    d = mdg.Domain(*box)
    for k in range(3):
        if per[k]:
            d.set_periodic(k, True)
    s = mdg.System(H.ctx(), d, atoms)
    mdg.VerletList(s).update(-1.0)
    sol = make(precision)
    sol.prepare(s)
    sol.stages(s)
    f = s.forces()
    s.close()
    return f


def _check(atoms, box, make, per=(1, 1, 1)):
    m, f = (_forces(atoms, box, make, p, per) for p in ("mixed", "fp64"))
    assert np.linalg.norm(m - f) <= 1e-5 * np.linalg.norm(f)


def _lj(p):
    return lambda prec: mdg.Single(mdg.LJsCut(p["a"], p["s"], p["rcut"]), periodic=True, precision=prec)


def _eam(p):
    t = p["tables"]
    return lambda prec: mdg.Single(mdg.EAM(t["rcut"], t["Femb"], t["Rho"], t["Vpar"], t["Nr1"], t["dr"], t["Nrh1"],
                                           t["drh"]), periodic=True, precision=prec)


@pytest.mark.parametrize("n", [2, 31, 32, 33, 63, 65, 255, 257])
def test_block_remainders(n):
    """An open cluster of n atoms (32 atoms a block, lists from empty up)."""
    atoms, box, _, p = W.lj_argon_fcc(ncell=5, jitter=0.02)
    _check(atoms[:n].copy(), box, _lj(p), per=(0, 0, 0))


@pytest.mark.parametrize("rc_sigma", [1.2, 1.6, 1.9, 2.5, 3.0, 3.6])
def test_list_lengths(rc_sigma):
    """Rounds of eight groups: lists of about 14 to 220 entries."""
    atoms, box, _, p = W.lj_argon_fcc(ncell=8, jitter=0.02)
    rc = rc_sigma * p["s"]
    atoms["rcut"], atoms["rns"] = rc, rc + 0.03
    _check(atoms, box, _lj(dict(p, rcut=rc)))


@pytest.mark.parametrize("n", [23999, 24000])
def test_rule_edge_lj(n):
    atoms, box, _, p = W.lj_argon_fcc(ncell=19, jitter=0.02)
    _check(atoms[:n].copy(), box, _lj(p))


@pytest.mark.parametrize("n", [29999, 30000, 44999, 45000])
def test_rule_edge_eam(n):
    atoms, box, _, p = W.eam_cu_fcc(ncell=23)
    _check(atoms[:n].copy(), box, _eam(p))


def test_multi():
    atoms, box, _, p = W.eam_nial_b2(ncell=12)
    rng = np.random.default_rng(1)
    atoms["r"] += rng.uniform(-0.004, 0.004, (len(atoms), 3))

    def make(prec):
        s = mdg.Multi(2, periodic=True, precision=prec)
        for (i, j), t in p["tables"].items():
            s.add_potential(i, j, mdg.EAM(t["rcut"], t["Femb"], t["Rho"], t["Vpar"], t["Nr1"], t["dr"], t["Nrh1"],
                                          t["drh"]))
        return s
    _check(atoms, box, make)

"""The FP64 force stages at the edges of their launch rule (lanes per atom by
system size), list lengths (the 64-entry turns of a lane, remainders) and
image rule (boxes of 2 rns and below, coordinates far from the origin),
against the CPU oracle.

Tolerance: both sides evaluate a pair in FP64 with a handful of roundings and
sum at most ~350 pairs in different orders; forces on a jittered lattice are
about a tenth of the sum of their terms' magnitudes, so 1e-10 of the largest
force leaves more than five orders of magnitude over 350 * 2^-53 * 10."""
from __future__ import annotations

import numpy as np
import pytest

import mdcraft_gb300 as mdg
from mdcraft_gb300 import workloads as W
from oracle import mdref as R

pytestmark = pytest.mark.gpu
TOL = 1e-10


def _oracle(atoms, box, per, make):
    a = np.zeros(len(atoms), dtype=R.ATOM_DTYPE)
    a.view(np.uint8)[:] = np.ascontiguousarray(atoms).view(np.uint8)
    d = R.Domain(*box)
    for k in range(3):
        if per[k]:
            d.set_periodic(k, True)
    nl = R.VerletList(a, d, threads=R.hardware_threads())
    nl.update(-1.0)
    s = R.Solver(make(R), periodic=d, threads=R.hardware_threads())
    s.prepare(a)
    s.stages(a, nl)
    s.virials(a, nl)
    return a


def _engine(atoms, box, per, make):
    from tests import gpu_helpers as H
    d = mdg.Domain(*box)
    for k in range(3):
        if per[k]:
            d.set_periodic(k, True)
    s = mdg.System(H.ctx(), d, atoms)
    mdg.VerletList(s).update(-1.0)
    sol = mdg.Single(make(mdg), periodic=True, precision="fp64")
    sol.prepare(s)
    sol.stages(s)
    sol.virials(s)
    out = s.download()
    s.close()
    return out


def _check(atoms, box, make, per=(1, 1, 1)):
    o, g = _oracle(atoms, box, per, make), _engine(atoms, box, per, make)
    for k in ("f", "V", "Ep", "Em", "nc"):
        big = np.abs(o[k]).max()
        assert np.abs(g[k] - o[k]).max() <= TOL * max(big, 1e-300), k


def _lj(p):
    return lambda M: M.LJsCut(p["a"], p["s"], p["rcut"])


def _eam(p):
    t = p["tables"]
    return lambda M: M.EAM(t["rcut"], t["Femb"], t["Rho"], t["Vpar"], t["Nr1"], t["dr"], t["Nrh1"], t["drh"])


@pytest.mark.parametrize("n", [12499, 12500, 12501])
def test_lanes_rule_edge(n):
    atoms, box, _, p = W.eam_cu_fcc(ncell=15)
    _check(atoms[:n].copy(), box, _eam(p))


@pytest.mark.parametrize("rc_sigma", [1.3, 2.5, 3.4, 4.2])
@pytest.mark.parametrize("ncell", [10, 15])
def test_list_lengths(ncell, rc_sigma):
    """Lists of about 20 to 350 entries, with 32 lanes (4,000 atoms) and 4 (13,500)."""
    atoms, box, _, p = W.lj_argon_fcc(ncell=ncell, jitter=0.02)
    rc = rc_sigma * p["s"]
    atoms["rcut"], atoms["rns"] = rc, rc + 0.03
    _check(atoms, box, _lj(dict(p, rcut=rc)))


@pytest.mark.parametrize("edge", [1.99, 2.0, 2.01])
def test_image_rule_edge(edge):
    """A box of about 2 rns: above it images come from FP32 signs, below from
    the reference's test."""
    atoms, box, _, p = W.lj_argon_fcc(ncell=4, jitter=0.02)
    atoms["rns"] = (box[1] - box[0]) / edge
    _check(atoms, box, _lj(p))


@pytest.mark.parametrize("skin", [-0.02, 0.0])
def test_list_radius_at_or_below_the_cutoff(skin):
    """rns at or below the cutoff: a pair can count raw and as a ghost."""
    atoms, box, _, p = W.lj_argon_fcc(ncell=5, jitter=0.02)
    atoms["rns"] = p["rcut"] + skin
    _check(atoms, box, _lj(p))


@pytest.mark.parametrize("shift", [-4000.0, 50.0, 1e5])
def test_box_far_from_the_origin(shift):
    """The FP32 screen's threshold grows with the coordinates."""
    atoms, box, _, p = W.eam_cu_fcc(ncell=5)
    atoms["r"] += shift
    _check(atoms, tuple(b + shift for b in box), _eam(p), per=(1, 1, 0))


def test_cutoff_past_the_table():
    """Pairs beyond the last interval contribute nothing (N1 >= Nr1); those in
    it read the padded knot."""
    atoms, box, _, p = W.eam_cu_fcc(ncell=5)
    t = dict(p["tables"])
    n = 700
    t.update(Rho=t["Rho"][:4200:6], Vpar=t["Vpar"][:4200:6], Nr1=n, dr=t["dr"] * 6)
    assert n * t["dr"] < t["rcut"]
    _check(atoms, box, _eam(dict(tables=t)))


def test_uneven_masses_step():
    """One step with masses of many magnitudes: the division by the mass from
    its reciprocal equals the FP64 division bit for bit."""
    from tests import gpu_helpers as H
    atoms, box, _, p = W.lj_argon_fcc(ncell=5, jitter=0.02)
    rng = np.random.default_rng(3)
    atoms["m"] = 10.0 ** rng.uniform(-3, 5, len(atoms))
    d = mdg.Domain(*box)
    for k in range(3):
        d.set_periodic(k, True)
    s = mdg.System(H.ctx(), d, atoms)
    mdg.VerletList(s).update(-1.0)
    sol = mdg.Single(_lj(p)(mdg), periodic=True, precision="fp64")
    sol.prepare(s)
    sol.stages(s)
    dt = 0.002
    f0, v0, r0 = s.forces(), s.velocities(), s.positions()
    mdg.Verlet(sol).make_step(s, dt)
    f1, m = s.forces(), atoms["m"][:, None]
    v = v0 + (f0 / m) * dt * 0.5
    assert np.array_equal(s.positions(), r0 + v * dt)
    assert np.array_equal(s.velocities(), v + (f1 / m) * 0.5 * dt)
    s.close()

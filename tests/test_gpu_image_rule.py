"""FP64 forces where FP32 coordinates cannot tell which image of a pair is in
range: an edge just above twice the list radius, a thin skin, and coordinates
so large that one FP32 step is longer than the skin.

Tolerance: as in test_gpu_forces64, and the oracle's ghosts sit at r_i + d, so
at coordinates X they are off by half an FP64 step there. LJ forces change by at
most 14 / r of themselves a unit of length, r >= 0.38 nm here: on forces of a
tenth of their terms' sum, less than 1,000 steps. A pair at the cutoff taken or
missed is more than 1e-4 of the largest force."""
from __future__ import annotations

import numpy as np
import pytest

from mdcraft_gb300 import workloads as W
from tests.test_gpu_forces64 import TOL, _engine, _lj, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skin", [0.001, 0.01])
@pytest.mark.parametrize("shift", [0.0, 3e4, -1e5, 1e6])
def test_thin_skin_far_from_the_origin(shift, skin):
    _, _, _, p = W.lj_argon_fcc(ncell=4)
    atoms = W.lj_argon_fcc(ncell=4)[0][:64].copy()
    rns = p["rcut"] + skin
    L = 2.0 * rns * 1.0001
    rng = np.random.default_rng(7)
    site = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    r = (site + 0.5) * (L / 4) + rng.uniform(-0.02, 0.02, (64, 3))
    # pairs two sites apart along an axis lie within a few hundredths of rc
    d = np.abs(r[:, None, 0] - r[None, :, 0])
    assert ((d > L / 2 - 0.03) & (d < p["rcut"])).any()
    atoms["r"] = r + shift
    atoms["rns"] = rns
    args = atoms, (shift, shift + L) * 3, (1, 1, 1), _lj(p)
    o, g = _oracle(*args), _engine(*args)
    tol = TOL + 1000.0 * np.spacing(abs(shift))
    for k in ("f", "V", "Ep"):
        assert np.abs(g[k] - o[k]).max() <= tol * np.abs(o[k]).max(), k

"""Records up and down on both sides of the line between the pinned staging and
a copy straight from the caller's memory (1,500 atoms), and totals of few parts."""
from __future__ import annotations

import numpy as np
import pytest

import mdcraft_gb300 as mdg
from tests import gpu_helpers as H

pytestmark = pytest.mark.gpu


def _system(n):
    rng = np.random.default_rng(n)
    a = mdg.new_atoms(n)
    for f in ("r", "v", "f"):
        a[f] = rng.uniform(0.0, 5.0, (n, 3))
    a["m"], a["rcut"], a["rns"] = rng.uniform(1.0, 2.0, n), 0.9, 1.0
    a["uid"], a["tag"] = np.arange(n) + 7, 1
    a["Ep"], a["Em"] = rng.normal(size=n), rng.normal(size=n)
    return mdg.System(H.ctx(), mdg.Domain(0, 5, 0, 5, 0, 5), a), a


@pytest.mark.parametrize("n", [1, 33, 1499, 1500, 1501, 4000])
def test_records_round_trip(n):
    s, a = _system(n)
    b = a[::-1].copy()
    s.upload(b)
    got = s.download()
    for f in ("r", "v", "f", "m", "rcut", "rns", "Ep", "Em", "uid", "kind", "tag"):
        assert np.array_equal(got[f], b[f]), f
    s.close()


@pytest.mark.parametrize("n", [1, 255, 256, 257, 600, 8192, 8193, 40000, 70000])
def test_totals_of_any_number_of_parts(n):
    """1 to 274 parts of 256 atoms; FP64 sums of n terms of about one, so 1e-12 of
    the sum of their sizes is more than their roundings."""
    s, a = _system(n)
    t = s.measure()
    m, v = a["m"], a["v"]
    com = (m[:, None] * v).sum(0) / m.sum()
    for k, want, size in (("Ep", a["Ep"].sum(), np.abs(a["Ep"]).sum()), ("Em", a["Em"].sum(), np.abs(a["Em"]).sum()),
                          ("KE", 0.5 * (m[:, None] * (v - com) ** 2).sum(), 0.5 * (m[:, None] * v ** 2).sum())):
        assert abs(t[k] - want) <= 1e-12 * size, k
    assert np.abs(t["vcom"] - com).max() <= 1e-12 * 5.0
    s.close()

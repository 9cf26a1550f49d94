"""Runs of more steps than one launch of a grid's team takes (a few
milliseconds): the same bits as the loop that launches every pass, and no
launch that holds the GPU for the whole run."""
from __future__ import annotations

import pytest

from tests import gpu_helpers as H
from tests.test_gpu_team import LANGEVIN, _check, _Run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,precision,steps,least", [("lj", 13500, "fp64", 250, 3), ("eam", 8788, "fp64", 200, 3),
                                                          ("lj", 4000, "mixed", 1500, 3), ("lj", 62500, "mixed", 400, 2)])
def test_launches_are_bounded(kind, n, precision, steps, least):
    """250 FP64 steps of 13,500 atoms take some 15 ms: not one launch."""
    r = _Run(kind, n, precision=precision)
    r.steps(2, False)
    before = H.ctx().launches()
    r.steps(steps, False)
    assert least <= H.ctx().launches() - before <= 40
    r.sys.close()


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("kind", ["lj", "eam"])
def test_same_bits_over_launches(kind, precision):
    """Stops at any step: with flipped buffers, at a rebuild, after one."""
    _check(precision, [700], kind, 2916, T=900.0, rns=lambda rc: rc + 0.01)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_thermostat_calls_over_launches(precision):
    _check(precision, [500], "eam", 2916, thermo=[LANGEVIN], tag0=7)

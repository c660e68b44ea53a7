"""Conversion switched off in mid-run: what the last step with it left on the device (marks of
sites near an interstitial that has since recombined; interstitials that the host has not
counted yet) must not change the steps that follow.  Against runs in which nothing is left
over, bitwise."""
from __future__ import annotations

import numpy as np
import pytest

import misa_b200 as mb
from scenarios import A0, MASS, make

pytestmark = pytest.mark.gpu
FIELDS = ("id", "type", "x", "v", "f", "rho", "df")
CELLS = (8, 7, 9)


def _sim(sc, precision):
    return mb.Sim(sc.cells, sc.tables, lattice_const=A0, mass=MASS, dt=1.0, cutoff=sc.cutoff, stencil_skin=sc.skin,
                  precision=precision, max_interstitials=8)


def _same(a, b):
    for k in FIELDS:
        assert np.array_equal(a[0][k], b[0][k]), k
        assert np.array_equal(a[1][k], b[1][k]), k


@pytest.mark.parametrize("precision", [mb.MB_PREC_FP64, mb.MB_PREC_MIXED])
@pytest.mark.parametrize("steps_before", [0, 1])  # the last step's marks: of either buffer
def test_off_after_the_last_recombination(precision, steps_before):
    sc = make(cells=CELLS, temperature=300.0, seed=131, n_itl=1)
    site = ((4 * CELLS[1]) + 3) * 2 * CELLS[0] + 6
    ideal = mb.lattice.bcc_box(CELLS, A0)["x"][site]
    sc.box["type"][site] = -1
    sc.itl["x"][0] = ideal + np.array([0.12, -0.07, 0.05])
    sc.itl["v"][0] = 0.0
    out = {}
    for off in (False, True):
        with _sim(sc, precision) as sim:
            sim.upload(sc.box, sc.itl)
            if steps_before:  # the interstitial stays until the step before conversion goes off
                sim.run(steps_before - 1)
            sim.set_conversion(0.7, 0.35)
            sim.run(min(steps_before, 1))
            assert sim.conversion_stats()["n_itl"] == 0
            if off:
                sim.set_conversion(0.0, 0.0)
            sim.run(6)
            out[off] = sim.download()
            if off:  # and on again: nothing of the old marks is left
                sim.set_conversion(0.7, 0.35)
            sim.run(3)
            out[off, "on again"] = sim.download()
    _same(out[True], out[False])
    _same(out[True, "on again"], out[False, "on again"])


def test_off_before_the_host_has_counted_the_interstitials():
    sc = make(cells=CELLS, temperature=300.0, seed=132)
    site = ((4 * CELLS[1]) + 3) * 2 * CELLS[0] + 6
    sc.box["x"][site] = mb.lattice.bcc_box(CELLS, A0)["x"][site] + np.array([0.55, 0.35, 0.0])
    out = {}
    for counted in (True, False):
        with _sim(sc, mb.MB_PREC_FP64) as sim:
            sim.upload(sc.box)
            sim.set_conversion(0.6, 0.3)
            sim.time_steps(1)  # steps without a synchronisation of the host's count
            if counted:
                sim.sync()
            sim.set_conversion(0.0, 0.0)
            sim.run(5)
            out[counted] = sim.download()
    assert len(out[True][1]) == 1
    _same(out[True], out[False])

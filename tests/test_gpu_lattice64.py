"""The two kinds of one-type FP64 lattice passes (shell windows for large launches, items
split over warps for small ones) against the oracle and bitwise against each other: ragged
rows, the smallest box, 5 and 6 shells inside the cutoff, coarse and fine tables, and
displacements that put many pairs outside their shell's table window.

Tolerances are the FP64 path's: forces within 1e-10 of the largest, rho within 1e-12."""
from __future__ import annotations

import numpy as np
import pytest

import misa_b200 as mb
from oracle import oracle as orc
from scenarios import A0, MASS, make, rel_err

pytestmark = pytest.mark.gpu

CASES = {
    "smallest": dict(cells=(5, 5, 5)),
    "rows_run_on": dict(cells=(33, 6, 5), vacancy=0.02),
    "full_rows": dict(cells=(32, 5, 7), n_itl=2, vacancy=0.01),
    "ragged_plane": dict(cells=(7, 9, 6), n_itl=3),
    "far_pairs": dict(cells=(9, 8, 7), vacancy=0.02, jitter=0.35),
    "six_shells": dict(cells=(8, 6, 7), cutoff=5.8, skin=0.5, jitter=0.1),
    "wide_skin": dict(cells=(8, 7, 6), skin=1.3, jitter=0.2),
    "coarse_table": dict(cells=(6, 7, 8), nr=1200, jitter=0.1),
    "fine_table": dict(cells=(6, 7, 8), nr=40000),
}


def _scenario(cells, cutoff=5.6, skin=0.7, nr=5000, **kw):
    sc = make(cells=cells, seed=61, tables=mb.potential.fe_analytic(nr=nr, cutoff=cutoff, rho_max=400.0), skin=skin, **kw)
    sc.cutoff = cutoff
    sc.ghost = mb.lattice.ghost_for_reach(A0, cutoff + skin)
    return sc


def _run(sc, nsteps, energy_every):
    with mb.Sim(sc.cells, sc.tables, lattice_const=A0, mass=MASS, dt=1.0, cutoff=sc.cutoff, stencil_skin=sc.skin,
                max_interstitials=max(1, sc.itl.shape[0])) as sim:
        sim.upload(sc.box, sc.itl if sc.itl.shape[0] else None)
        sim.run(nsteps, energy_every)
        return *sim.download(), sim.energies()


@pytest.mark.parametrize("name", CASES)
def test_both_lattice_passes_match_the_oracle_and_each_other(name, monkeypatch):
    sc = _scenario(**CASES[name])
    got = {}
    for kind, items in (("shell", "0"), ("split", "1000000")):
        monkeypatch.setenv("MB_SPLIT_RHO_ITEMS", items)
        monkeypatch.setenv("MB_SPLIT_FORCE_ITEMS", items)
        got[kind] = _run(sc, 3, 1)
    ext = sc.ext().view(orc.ATOM)
    itl = sc.itl.view(orc.ATOM).copy()
    even, odd = sc.stencil()
    e = orc.md_run(sc.orc_pot(), sc.orc_domain(), ext, itl if itl.shape[0] else None, even, odd, sc.md_params(), 3)
    ref = mb.lattice.ext_to_box(ext, sc.cells, sc.ghost)
    live = ref["type"] >= 0
    for box, il, en in got.values():
        assert rel_err(box["f"][live], ref["f"][live]) < 1e-10
        assert rel_err(box["rho"][live], ref["rho"][live]) < 1e-12
        assert rel_err(box["df"][live], ref["df"][live]) < 1e-12
        assert np.max(np.abs(en[:, 1:] - e)) / live.sum() < 1e-12
        if itl.shape[0]:
            assert rel_err(il["f"], itl["f"]) < 1e-10
    for k in ("x", "v", "f", "rho", "df"):
        assert np.array_equal(got["shell"][0][k], got["split"][0][k]), k

"""FP64 lattice passes with two and three atom types, both kinds (shell windows, items split
over warps) against the oracle and bitwise against each other: split tables that fit shared
memory and that do not, windows in several copies and in one, ragged rows, vacant sites,
interstitials, five and six shells, and pairs far outside their shell's window.

Tolerances are the FP64 path's: forces within 1e-10 of the largest, rho within 1e-12."""
from __future__ import annotations

import numpy as np
import pytest

import misa_b200 as mb
from oracle import oracle as orc
from scenarios import A0, MASS, make, rel_err

pytestmark = pytest.mark.gpu

CASES = {
    "two": dict(n_types=2, cells=(33, 5, 6), vacancy=0.02),
    "two_fine_table": dict(n_types=2, cells=(7, 9, 6), nr=5000, n_itl=2),
    "three": dict(n_types=3, cells=(6, 7, 8), vacancy=0.01, n_itl=3),
    "three_fine_table": dict(n_types=3, cells=(9, 6, 5), nr=5000, jitter=0.1),
    "three_coarse_table": dict(n_types=3, cells=(6, 7, 5), nr=700),
    "far_pairs": dict(n_types=3, cells=(9, 8, 7), vacancy=0.02, nr=5000, jitter=0.35),
    "six_shells": dict(n_types=2, cells=(8, 6, 7), cutoff=5.8, skin=0.5, jitter=0.1),
    "too_fine_for_windows": dict(n_types=3, cells=(6, 7, 8), nr=20000),
}


def _run(sc, cutoff, nsteps):
    with mb.Sim(sc.cells, sc.tables, lattice_const=A0, mass=MASS, dt=1.0, cutoff=cutoff, stencil_skin=sc.skin,
                max_interstitials=max(1, sc.itl.shape[0])) as sim:
        sim.upload(sc.box, sc.itl if sc.itl.shape[0] else None)
        sim.run(nsteps, 1)
        return *sim.download(), sim.energies()


@pytest.mark.parametrize("name", CASES)
def test_alloy_passes_match_the_oracle_and_each_other(name, monkeypatch):
    kw = dict(CASES[name])
    nr, cutoff = kw.pop("nr", 2000), kw.pop("cutoff", 5.6)
    sc = make(seed=71, tables=mb.potential.alloy_analytic(kw["n_types"], nr=nr, cutoff=cutoff, rho_max=400.0),
              **{"skin": 0.7, **kw})
    sc.cutoff = cutoff
    sc.ghost = mb.lattice.ghost_for_reach(A0, cutoff + sc.skin)
    got = {}
    for kind, items in (("shell", "0"), ("split", "1000000")):
        monkeypatch.setenv("MB_SPLIT_RHO_ITEMS", items)
        monkeypatch.setenv("MB_SPLIT_FORCE_ITEMS", items)
        got[kind] = _run(sc, cutoff, 3)
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

"""Mixed-precision steps whose items are split over a CTA give the bits of the warp-per-item
kernels: 7 and 8 built-in shells, ragged and smallest lattices, vacant sites, interstitials,
conversion, and several lattices (more than a warp's width of them) with different targets."""
from __future__ import annotations

import numpy as np
import pytest

import misa_b200 as mb
from oracle import oracle as orc
from scenarios import A0, MASS, make

pytestmark = pytest.mark.gpu
FIELDS = ("type", "x", "v", "f", "rho", "df")

CASES = {
    "smallest": dict(cells=(5, 5, 5)),
    "ragged": dict(cells=(33, 6, 7), vacancy=0.02),
    "interstitials": dict(cells=(11, 9, 8), vacancy=0.01, n_itl=4),
    "eight_shells": dict(cells=(9, 12, 7), skin=1.3, temperature=900.0, vacancy=0.01),
    "conversion": dict(cells=(12, 11, 13), n_itl=3, skin=1.3, temperature=1200.0),
}


@pytest.mark.parametrize("name", CASES)
def test_split_items_give_the_same_bits(name, monkeypatch):
    sc = make(seed=101, **{"temperature": 600.0, **CASES[name]})
    got = {}
    for items in ("0", "1000000"):
        monkeypatch.setenv("MB_MX_ONE_ITEMS", items)
        with mb.Sim(sc.cells, sc.tables, lattice_const=A0, mass=MASS, dt=1.0, cutoff=sc.cutoff, stencil_skin=sc.skin,
                    precision=mb.MB_PREC_MIXED, max_interstitials=64) as sim:
            sim.upload(sc.box, sc.itl if sc.itl.shape[0] else None)
            if name == "conversion":
                sim.set_conversion(sc.skin, 0.5 * sc.skin)
            sim.run(40, 15)
            got[items] = sim.download()
    for a, b in zip(got["0"], got["1000000"]):
        for k in FIELDS:
            assert np.array_equal(a[k], b[k]), k


def test_split_items_of_many_lattices_give_the_same_bits(monkeypatch):
    cells = [(5 + k % 4, 5 + k % 3, 5 + k % 5) for k in range(37)] + [(17, 9, 12)]
    scs = [make(cells=c, seed=102 + k, vacancy=0.01 * (k % 3)) for k, c in enumerate(cells)]
    got = {}
    for items in ("0", "1000000"):
        monkeypatch.setenv("MB_MX_ONE_ITEMS", items)
        with mb.Ensemble(scs[0].tables, lattice_const=A0, mass=MASS, dt=1.0, cutoff=scs[0].cutoff,
                         stencil_skin=scs[0].skin) as ens:
            slots = [ens.add(sc.cells, sc.box, None, 20 + k % 7) for k, sc in enumerate(scs)]
            while ens.advance(10):
                pass
            got[items] = [ens.download(s)[0] for s in slots]
    for a, b in zip(got["0"], got["1000000"]):
        for k in FIELDS:
            assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("n_itl", [64, 65])
def test_interstitials_as_a_list_and_in_cells_match_the_oracle(n_itl):
    # up to 64 interstitials are walked as a list, more through the cell list
    sc = make(cells=(16, 15, 14), temperature=900.0, vacancy=0.01, n_itl=n_itl, seed=103, jitter=0.1)
    with mb.Sim(sc.cells, sc.tables, lattice_const=A0, mass=MASS, dt=1.0, cutoff=sc.cutoff, stencil_skin=sc.skin,
                precision=mb.MB_PREC_MIXED, max_interstitials=n_itl) as sim:
        sim.upload(sc.box, sc.itl)
        sim.run(0)
        box, itl = sim.download()
    even, odd = sc.stencil()
    ext, il = sc.ext().view(orc.ATOM), sc.itl.view(orc.ATOM).copy()
    orc.compute_forces(sc.orc_pot(), sc.orc_domain(), ext, il, even, odd, sc.md_params())
    ref = mb.lattice.ext_to_box(ext, sc.cells, sc.ghost)
    live = ref["type"] >= 0
    got = np.concatenate([box["f"][live], itl["f"]])
    want = np.concatenate([ref["f"][live], il["f"]])
    assert np.sqrt(np.mean((got - want) ** 2)) < 1e-6 * np.sqrt(np.mean(want**2))
    got, want = np.concatenate([box["rho"][live], itl["rho"]]), np.concatenate([ref["rho"][live], il["rho"]])
    assert np.sqrt(np.mean((got - want) ** 2)) < 1e-6 * np.sqrt(np.mean(want**2))

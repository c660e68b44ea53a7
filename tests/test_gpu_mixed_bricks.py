"""The brick walk of one mixed-precision lattice, which only large lattices take by themselves
(MB_MX_BRICKS asks for it here): 7 and 8 built-in shells, ragged bricks, energy steps,
interstitials, conversion, outer-entry masks and chained kernels.  The walk must not change a
bit of the state; energies are summed in another order."""
from __future__ import annotations

import numpy as np
import pytest

import misa_b200 as mb
from oracle import oracle as orc
from scenarios import A0, MASS, make

pytestmark = pytest.mark.gpu
FIELDS = ("type", "x", "v", "f", "rho", "df")
CASES = {
    "seven_shells": dict(cells=(40, 13, 11), vacancy=0.01, jitter=0.1),
    "eight_shells": dict(cells=(33, 10, 17), vacancy=0.01, skin=1.3, temperature=900.0, jitter=0.1),
    "interstitials": dict(cells=(64, 9, 10), vacancy=0.01, n_itl=5),
    "narrow": dict(cells=(7, 6, 9), n_itl=2, skin=1.3),
    "conversion": dict(cells=(20, 21, 9), n_itl=4, skin=1.3, temperature=1200.0),
}


def _run(sc, bricks, monkeypatch, conversion=False, steps=24, every=5):
    monkeypatch.setenv("MB_MX_BRICKS", "1" if bricks else "0")
    monkeypatch.setenv("MB_MX_ONE_ITEMS", "0")
    with mb.Sim(sc.cells, sc.tables, lattice_const=A0, mass=MASS, dt=1.0, cutoff=sc.cutoff, stencil_skin=sc.skin,
                precision=mb.MB_PREC_MIXED, max_interstitials=64) as sim:
        sim.upload(sc.box, sc.itl if sc.itl.shape[0] else None)
        if conversion:
            sim.set_conversion(sc.skin, 0.5 * sc.skin)
        sim.run(steps, every)
        assert sim.pass_kinds() == (("bricks",) * 2 if bricks else ("linear",) * 2)
        return *sim.download(), sim.energies()


def _same(a, b):
    for x, y in zip(a[:2], b[:2]):
        for k in FIELDS:
            assert np.array_equal(x[k], y[k]), k
    # sums of some 10^4 terms of one sign: 10^4 roundings of 1.1e-16 at most (the order is the
    # walk's, and no fixed one for the interstitials' part)
    assert np.array_equal(a[2][:, 0], b[2][:, 0])
    assert np.max(np.abs(a[2][:, 1:] / b[2][:, 1:] - 1.0)) < 2e-12


@pytest.mark.parametrize("name", CASES)
def test_bricks_give_the_bits_of_linear_items(name, monkeypatch):
    sc = make(seed=151, **{"temperature": 600.0, **CASES[name]})
    linear = _run(sc, False, monkeypatch, name == "conversion")
    bricks = _run(sc, True, monkeypatch, name == "conversion")
    _same(bricks, linear)


@pytest.mark.parametrize("name", ["seven_shells", "eight_shells", "interstitials"])
@pytest.mark.parametrize("switch", ["MB_OUTER_MASKS", "MB_CHAIN"])
def test_bricks_without_masks_and_without_chains_give_the_same_bits(name, switch, monkeypatch):
    sc = make(seed=152, **{"temperature": 900.0, **CASES[name]})
    on = _run(sc, True, monkeypatch)
    monkeypatch.setenv(switch, "0")
    off = _run(sc, True, monkeypatch)
    _same(on, off)


@pytest.mark.parametrize("name", ["seven_shells", "eight_shells", "interstitials"])
def test_brick_forces_match_the_oracle(name, monkeypatch):
    sc = make(seed=153, **{"temperature": 600.0, **CASES[name]})
    box, itl, _ = _run(sc, True, monkeypatch, steps=0, every=0)
    even, odd = sc.stencil()
    ext, il = sc.ext().view(orc.ATOM), sc.itl.view(orc.ATOM).copy()
    orc.compute_forces(sc.orc_pot(), sc.orc_domain(), ext, il, even, odd, sc.md_params())
    ref = mb.lattice.ext_to_box(ext, sc.cells, sc.ghost)
    live = ref["type"] >= 0
    for k in ("f", "rho"):
        got, want = np.concatenate([box[k][live], itl[k]]), np.concatenate([ref[k][live], il[k]])
        assert np.sqrt(np.mean((got - want) ** 2)) < 1e-6 * np.sqrt(np.mean(want**2)), k

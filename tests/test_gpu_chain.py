"""Steps whose kernels start while the one before drains give the same bits as steps whose
kernels run one by one: both kinds of FP64 pass, one and several types, interstitials,
conversion, bricks, linear items and several lattices of the mixed path."""
from __future__ import annotations

import numpy as np
import pytest

import misa_b200 as mb
from scenarios import A0, MASS, make

pytestmark = pytest.mark.gpu

CASES = {
    "split": dict(cells=(9, 7, 8), vacancy=0.01),
    "shell": dict(cells=(33, 36, 41), vacancy=0.01),
    "shell_itl": dict(cells=(33, 36, 41), vacancy=0.01, n_itl=12),
    "conversion": dict(cells=(20, 21, 19), n_itl=4, temperature=1200.0, conv=True),
    "alloy": dict(cells=(19, 12, 14), n_types=3, n_itl=3),
    "mixed": dict(cells=(20, 9, 11), vacancy=0.01, mixed=True),
    "mixed_bricks": dict(cells=(64, 48, 48), vacancy=0.01, mixed=True),
    "mixed_itl": dict(cells=(33, 30, 21), n_itl=9, mixed=True),
    "mixed_conversion": dict(cells=(20, 21, 19), n_itl=4, temperature=1200.0, mixed=True, conv=True),
}


def _run(sc, mixed, conv):
    kw = dict(lattice_const=A0, mass=MASS, dt=1.0, cutoff=sc.cutoff, stencil_skin=sc.skin)
    with mb.Sim(sc.cells, sc.tables, precision=mb.MB_PREC_MIXED if mixed else mb.MB_PREC_FP64,
                max_interstitials=64 if conv else max(1, sc.itl.shape[0]), **kw) as sim:
        sim.upload(sc.box, sc.itl if sc.itl.shape[0] else None)
        if conv:
            sim.set_conversion(sc.skin, 0.5 * sc.skin)
        sim.run(60, 25)
        return sim.download()


@pytest.mark.parametrize("name", CASES)
def test_chained_steps_give_the_same_bits(name, monkeypatch):
    kw = dict(CASES[name])
    mixed, conv = kw.pop("mixed", False), kw.pop("conv", False)
    sc = make(seed=91, **{"temperature": 600.0, **kw})
    got = {}
    for chain in ("1", "0"):
        monkeypatch.setenv("MB_CHAIN", chain)
        got[chain] = [_run(sc, mixed, conv) for _ in range(2)]
    ref = got["0"][0]
    for box, itl in got["1"] + got["0"][1:]:
        for k in ("type", "x", "v", "f", "rho", "df"):
            assert np.array_equal(box[k], ref[0][k]), k
            assert np.array_equal(itl[k], ref[1][k]), k


def test_chained_ensemble_steps_give_the_same_bits(monkeypatch):
    scs = [make(cells=c, seed=92 + i, vacancy=0.01) for i, c in enumerate([(6, 7, 5), (17, 9, 12), (24, 22, 19)])]
    got = {}
    for chain in ("1", "0"):
        monkeypatch.setenv("MB_CHAIN", chain)
        with mb.Ensemble(scs[0].tables, lattice_const=A0, mass=MASS, dt=1.0, cutoff=scs[0].cutoff,
                         stencil_skin=scs[0].skin) as ens:
            slots = [ens.add(sc.cells, sc.box) for sc in scs]
            ens.run(60)
            got[chain] = [ens.download(s)[0] for s in slots]
    for a, b in zip(got["1"], got["0"]):
        for k in ("x", "v", "f", "rho", "df"):
            assert np.array_equal(a[k], b[k]), k

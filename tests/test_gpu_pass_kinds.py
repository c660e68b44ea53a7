"""Which kernels a lattice takes, where tests compare two kinds of pass by environment
variables alone: shell windows against split items wherever the plan applies, the row walk on
both sides where the tables are too fine for windows or the stencil is not built in."""
from __future__ import annotations

import pytest

import misa_b200 as mb
import test_gpu_alloy_lattice64 as alloy
import test_gpu_lattice64 as one_type
from scenarios import A0, MASS, make

pytestmark = pytest.mark.gpu


def _kinds(sc, monkeypatch, items, precision=mb.MB_PREC_FP64, a0=A0):
    for name in ("MB_SPLIT_RHO_ITEMS", "MB_SPLIT_FORCE_ITEMS"):
        if items is None:
            monkeypatch.delenv(name, raising=False)
        else:
            monkeypatch.setenv(name, items)
    with mb.Sim(sc.cells, sc.tables, lattice_const=a0, mass=MASS, dt=1.0, cutoff=sc.cutoff,
                stencil_skin=sc.skin, precision=precision) as sim:
        if precision == mb.MB_PREC_MIXED:
            sim.upload(sc.box)
        return sim.pass_kinds()


@pytest.mark.parametrize("name", one_type.CASES)
def test_kinds_of_the_one_type_cases(name, monkeypatch):
    sc = one_type._scenario(**one_type.CASES[name])
    rows = name == "fine_table"
    assert _kinds(sc, monkeypatch, "0") == (("rows",) * 2 if rows else ("shells",) * 2)
    assert _kinds(sc, monkeypatch, "1000000") == (("rows",) * 2 if rows else ("split",) * 2)


@pytest.mark.parametrize("name", alloy.CASES)
def test_kinds_of_the_alloy_cases(name, monkeypatch):
    kw = dict(alloy.CASES[name])
    nr, cutoff = kw.pop("nr", 2000), kw.pop("cutoff", 5.6)
    sc = make(seed=71, tables=mb.potential.alloy_analytic(kw["n_types"], nr=nr, cutoff=cutoff, rho_max=400.0), **kw)
    sc.cutoff = cutoff
    rows = name == "too_fine_for_windows"
    assert _kinds(sc, monkeypatch, "0") == (("rows",) * 2 if rows else ("shells",) * 2)
    assert _kinds(sc, monkeypatch, "1000000") == (("rows",) * 2 if rows else ("split",) * 2)


def test_kinds_by_size_and_stencil(monkeypatch):
    small, large = make(cells=(8, 8, 8)), make(cells=(48, 40, 44))
    assert _kinds(small, monkeypatch, None) == ("split", "split")
    assert _kinds(large, monkeypatch, None) == ("shells", "shells")
    assert _kinds(small, monkeypatch, None, a0=3.3) == ("rows", "rows")  # four shells inside the cutoff
    assert _kinds(small, monkeypatch, None, mb.MB_PREC_MIXED) == ("linear_split", "linear_split")
    assert _kinds(large, monkeypatch, None, mb.MB_PREC_MIXED) == ("linear", "linear")

"""Two box atoms at one point, and the undefined positions that follow: every kind of FP64
lattice pass (shell windows, split items, the row walk of tables too fine for windows) and
both kinds of hook pass, one type and three.

The coincident pair has no distance, and its force is undefined.  Its density term is undefined
too in one type (F' is then that of the last knot), and in several the density function's
last knot, where the oracle takes the first one (r = 0).  All else is the oracle's, with that
F'.  Tolerances are the FP64 path's: forces within 1e-10 of the largest, rho within 1e-12."""
from __future__ import annotations

import numpy as np
import pytest

import misa_b200 as mb
from oracle import oracle as orc
from scenarios import A0, MASS, make, rel_err

pytestmark = pytest.mark.gpu
CELLS = (7, 6, 6)
I = ((3 * 6) + 3) * 14 + 6  # box index of site (6, 3, 3), x doubled
J = I + 1                   # its neighbour half a cell up


def _scenario(n_types, fine=False):
    nr = {1: 40000 if fine else 5000, 3: 20000 if fine else 2000}[n_types]
    tables = mb.potential.fe_analytic(nr=nr, rho_max=400.0) if n_types == 1 else mb.potential.alloy_analytic(3, nr=nr)
    sc = make(cells=CELLS, seed=112, n_types=n_types, jitter=0.05, tables=tables)
    sc.box["x"][J] = sc.box["x"][I]
    return sc


def _expected(sc):
    pot, dom = sc.orc_pot(), sc.orc_domain()
    even, odd = sc.stencil()
    edge = [c * A0 for c in sc.cells]
    ext = sc.ext().view(orc.ATOM)
    orc.rho_pass(pot, dom, ext, even, odd, sc.cutoff)
    box = mb.lattice.ext_to_box(ext, sc.cells, sc.ghost)
    for a, b in ((I, J), (J, I)):
        f, last = sc.tables.f[box["type"][b]], sc.tables.drho * (sc.tables.F.shape[1] - 1)
        box["rho"][a] = box["rho"][a] + f[-1] - f[0] if sc.tables.n_types > 1 else np.nan
        box["df"][a] = pot.dF(int(box["type"][a]), box["rho"][a] if sc.tables.n_types > 1 else last)
    grid = ext.reshape(CELLS[2] + 2 * sc.ghost[2], CELLS[1] + 2 * sc.ghost[1], 2 * CELLS[0] + 2 * sc.ghost[0])
    inner = grid[sc.ghost[2]:-sc.ghost[2], sc.ghost[1]:-sc.ghost[1], sc.ghost[0]:-sc.ghost[0]]
    inner["df"] = box["df"].reshape(inner.shape)
    orc.ghost_fill(dom, ext, edge, 2)
    orc.force_pass(pot, dom, ext, even, odd, sc.cutoff)
    f = mb.lattice.ext_to_box(ext, sc.cells, sc.ghost)["f"]
    return box["rho"], box["df"], f


def _check(got, want):
    rho, df, f = want
    others = np.ones(len(rho), bool)
    others[[I, J]] = False
    defined = np.isfinite(rho)
    assert np.array_equal(np.isfinite(got["rho"]), defined)
    assert rel_err(got["rho"][defined], rho[defined]) < 1e-12
    assert rel_err(got["df"], df) < 1e-12
    assert rel_err(got["f"][others], f[others]) < 1e-10
    assert not np.isfinite(got["f"][[I, J]]).any()


@pytest.mark.parametrize("n_types", [1, 3])
@pytest.mark.parametrize("kind", ["shell", "split", "rows"])
def test_resident_passes_with_coincident_atoms(kind, n_types, monkeypatch):
    sc = _scenario(n_types, fine=kind == "rows")
    items = "1000000" if kind == "split" else "0"
    monkeypatch.setenv("MB_SPLIT_RHO_ITEMS", items)
    monkeypatch.setenv("MB_SPLIT_FORCE_ITEMS", items)
    with mb.Sim(sc.cells, sc.tables, lattice_const=A0, mass=MASS, dt=1.0, cutoff=sc.cutoff, stencil_skin=sc.skin) as sim:
        assert sim.pass_kinds() == ({"shell": "shells"}.get(kind, kind),) * 2
        sim.upload(sc.box)
        sim.run(0, 1)
        first = sim.download()[0]
        sim.run(2)  # both atoms now have undefined positions: no pair with them is inside the cutoff
        later = sim.download()[0]
    _check(first, _expected(sc))
    if kind == "rows" and n_types == 1:
        return  # masks a pair by a zero factor: its neighbours' forces become undefined too
    others = np.ones(len(sc.box), bool)
    others[[I, J]] = False
    for k in ("x", "v", "f", "rho", "df"):
        assert np.isfinite(later[k][others]).all(), k


@pytest.mark.parametrize("n_types", [1, 3])
@pytest.mark.parametrize("kind", ["split", "rows"])
def test_hook_passes_with_coincident_atoms(kind, n_types, monkeypatch):
    sc = _scenario(n_types)
    monkeypatch.setenv("MB_HOOK_SPLIT_ITEMS", "1000000" if kind == "split" else "0")
    dom = mb.lattice.domain(sc.cells, sc.ghost, (0, 0, 0))
    hooks = mb.Hooks(0)
    try:
        hooks.domain_init(dom)
        hooks.nei_offset_init(*mb.lattice.stencil_linear(A0, sc.reach, dom.ext_size_x, dom.ext_size_y))
        hooks.pot_init(sc.tables)
        ext = sc.ext()
        hooks.rho_calc(ext, sc.cutoff)
        orc.ghost_fill(sc.orc_domain(), ext.view(orc.ATOM), [c * A0 for c in sc.cells], 2)
        hooks.force_calc(ext, sc.cutoff)
    finally:
        mb.Hooks.clean()
    _check(mb.lattice.ext_to_box(ext, sc.cells, sc.ghost), _expected(sc))

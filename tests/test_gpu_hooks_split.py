"""The rho and force hooks by split items and by the row walk, against the oracle: ragged and
smallest boxes, one and three types, stencils in reverse order and with more entries than the
split items take, and slab counts that have to give the same bytes.

Tolerances are the FP64 path's: forces within 1e-10 of the largest, rho within 1e-12."""
from __future__ import annotations

import numpy as np
import pytest

import misa_b200 as mb
from oracle import oracle as orc
from scenarios import A0, make, rel_err

pytestmark = pytest.mark.gpu

CASES = {
    "smallest": dict(cells=(5, 5, 5)),
    "ragged": dict(cells=(33, 6, 7), vacancy=0.02),
    "reversed": dict(cells=(9, 7, 6), vacancy=0.01, backwards=True),
    "alloy": dict(cells=(8, 9, 7), vacancy=0.01, n_types=3),
    "full_runs": dict(cells=(9, 9, 9), reach=8.5),   # 228 entries or so
    "too_long": dict(cells=(11, 10, 10), reach=9.4),  # more than 256: row walk on both sides
}


@pytest.fixture(scope="module")
def hooks():
    h = mb.Hooks(0)
    yield h
    mb.Hooks.clean()


@pytest.mark.parametrize("name", CASES)
def test_hook_passes_match_the_oracle(hooks, name, monkeypatch):
    kw = dict(CASES[name])
    reach, backwards = kw.pop("reach", None), kw.pop("backwards", False)
    sc = make(seed=111, temperature=900.0, jitter=0.1, **kw)
    if reach:
        sc.ghost = mb.lattice.ghost_for_reach(A0, reach)
    dom = mb.lattice.domain(sc.cells, sc.ghost, (0, 0, 0))
    even, odd = mb.lattice.stencil_linear(A0, reach or sc.reach, dom.ext_size_x, dom.ext_size_y)
    if backwards:
        even, odd = even[::-1].copy(), odd[::-1].copy()
    hooks.domain_init(dom)
    hooks.nei_offset_init(even, odd)
    hooks.pot_init(sc.tables)
    odom = orc.make_domain(sc.cells, sc.ghost, (0, 0, 0))
    edge = [c * A0 for c in sc.cells]
    ref = sc.ext().view(orc.ATOM)
    orc.rho_pass(sc.orc_pot(), odom, ref, even, odd, sc.cutoff)
    orc.ghost_fill(odom, ref, edge, 2)
    orc.force_pass(sc.orc_pot(), odom, ref, even, odd, sc.cutoff)
    want = mb.lattice.ext_to_box(ref, sc.cells, sc.ghost)
    live = want["type"] >= 0
    for items in ("0", "1000000"):
        monkeypatch.setenv("MB_HOOK_SPLIT_ITEMS", items)
        out = []
        try:
            for batches in (1, 3):
                hooks.set_batches(batches)
                ext = sc.ext()
                hooks.rho_calc(ext, sc.cutoff)
                orc.ghost_fill(odom, ext.view(orc.ATOM), edge, 2)
                hooks.force_calc(ext, sc.cutoff)
                out.append(ext)
        finally:
            hooks.set_batches(1)
        assert out[0].tobytes() == out[1].tobytes()
        got = mb.lattice.ext_to_box(out[0], sc.cells, sc.ghost)
        assert rel_err(got["rho"][live], want["rho"][live]) < 1e-12
        assert rel_err(got["df"][live], want["df"][live]) < 1e-12
        assert rel_err(got["f"][live], want["f"][live]) < 1e-10


@pytest.mark.parametrize("n_types", [1, 3])
def test_degenerate_positions_as_in_the_row_walk(hooks, n_types, monkeypatch):
    # coincident atoms, infinite and undefined coordinates: finite where the row walk is finite
    sc = make(cells=(7, 6, 6), seed=112, n_types=n_types, jitter=0.05)
    dom = mb.lattice.domain(sc.cells, sc.ghost, (0, 0, 0))
    even, odd = mb.lattice.stencil_linear(A0, sc.reach, dom.ext_size_x, dom.ext_size_y)
    hooks.domain_init(dom)
    hooks.nei_offset_init(even, odd)
    hooks.pot_init(sc.tables)
    ext = sc.ext()
    mid = ext.shape[0] // 2 + 3
    ext["x"][mid] = ext["x"][mid + 1]
    ext["x"][mid + 40, 1] = np.inf
    ext["x"][mid - 40, 2] = np.nan
    got = {}
    for items in ("0", "1000000"):
        monkeypatch.setenv("MB_HOOK_SPLIT_ITEMS", items)
        e = ext.copy()
        hooks.rho_calc(e, sc.cutoff)
        # the pair that coincides has no finite df in one type: keep the force pass's own case apart
        e["df"] = np.where(np.isfinite(e["df"]), e["df"], 0.0)
        hooks.force_calc(e, sc.cutoff)
        got[items] = e
    for k, tol in (("rho", 1e-12), ("f", 1e-10)):
        a, b = got["0"][k], got["1000000"][k]
        fin = np.isfinite(a)
        assert np.array_equal(fin, np.isfinite(b)), k
        assert np.max(np.abs(a[fin] - b[fin])) <= tol * max(1.0, np.max(np.abs(a[fin]))), k

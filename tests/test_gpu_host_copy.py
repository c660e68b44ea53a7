"""Records that cross to the device and back through the shared pageable copies: sizes below
and above the threshold of the shared copy, before and after its slots are there, whole chunks and a short last one."""
from __future__ import annotations

import numpy as np
import pytest

import misa_b200 as mb
from scenarios import A0, MASS, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(6, 5, 7), (21, 21, 22), (32, 32, 32), (40, 41, 43), (56, 57, 55)])
@pytest.mark.parametrize("kind", ["fp64", "ensemble"])
def test_uploaded_records_come_back(cells, kind):
    sc = make(cells=cells, vacancy=0.01, seed=81)
    sc.box["f"] = np.random.default_rng(1).normal(size=sc.box["f"].shape)
    kw = dict(lattice_const=A0, mass=MASS, dt=1.0, cutoff=sc.cutoff, stencil_skin=sc.skin)
    if kind == "fp64":
        with mb.Sim(sc.cells, sc.tables, **kw) as sim:
            for _ in range(6):  # the page-locked slots come in on the way
                sim.upload(sc.box)
                got = sim.download()[0]
        fields, tol = ("id", "type", "x", "v", "f"), 0.0
    else:
        with mb.Ensemble(sc.tables, **kw) as ens:
            for _ in range(6):
                slot = ens.add(sc.cells, sc.box)
                got = ens.download(slot)[0]
                ens.remove(slot)
        # positions are kept as displacements from the ideal sites: one rounding each way
        fields, tol = ("id", "type", "x", "v"), 4e-14
    live = sc.box["type"] >= 0
    assert np.array_equal(got["id"], sc.box["id"]) and np.array_equal(got["type"], sc.box["type"])
    for k in fields[2:]:
        assert np.max(np.abs(got[k][live] - sc.box[k][live])) <= tol, k


@pytest.mark.parametrize("slabs", [1, 5])
@pytest.mark.parametrize("cells,n_itl", [((6, 7, 24), 0), ((9, 8, 27), 6)])
def test_host_steps_match_resident_steps(cells, n_itl, slabs, monkeypatch):
    # records in, drifted and given their ghost images by one kernel, kernels chained or one by one
    sc = make(cells=cells, vacancy=0.02, n_itl=n_itl, seed=82)
    kw = dict(lattice_const=A0, mass=MASS, dt=1.0, cutoff=sc.cutoff, stencil_skin=sc.skin, max_interstitials=8)
    with mb.Sim(sc.cells, sc.tables, **kw) as sim:
        sim.upload(sc.box, sc.itl if n_itl else None)
        sim.run(0)
        start = sim.download()
        sim.run(1)
        want = sim.download()
    got = {}
    for chain in ("1", "0"):
        monkeypatch.setenv("MB_CHAIN", chain)
        box, itl = start[0].copy(), start[1].copy()
        with mb.Sim(sc.cells, sc.tables, **kw) as sim:
            sim.set_host_slabs(slabs)
            sim.step_host(box, itl if n_itl else None)
        got[chain] = box, itl
    for k in ("id", "type", "x", "f", "rho", "df", "v"):
        assert np.array_equal(got["0"][0][k], got["1"][0][k]) and np.array_equal(got["0"][1][k], got["1"][1][k]), k
    live = want[0]["type"] >= 0
    assert np.array_equal(got["1"][0]["id"], want[0]["id"]) and np.array_equal(got["1"][0]["type"], want[0]["type"])
    # one drift from the same records: positions to the rounding of the half-step velocity,
    # forces to that of the positions
    assert np.max(np.abs(got["1"][0]["x"][live] - want[0]["x"][live])) < 1e-12
    assert np.max(np.abs(got["1"][0]["f"][live] - want[0]["f"][live])) < 1e-10 * np.max(np.abs(want[0]["f"][live]))
    if n_itl:
        assert np.max(np.abs(got["1"][1]["x"] - want[1]["x"])) < 1e-12
        assert np.array_equal(got["1"][1]["type"], want[1]["type"]) and np.array_equal(got["1"][1]["id"], want[1]["id"])

"""Records that cross to the device and back through the shared pageable copies: sizes below
and above the threshold of the shared copy, before and after its slots are there, whole chunks and a short last one."""
from __future__ import annotations

import numpy as np
import pytest

import misa_b200 as mb
from scenarios import A0, MASS, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(6, 5, 7), (21, 21, 22), (32, 32, 32), (40, 41, 43)])
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

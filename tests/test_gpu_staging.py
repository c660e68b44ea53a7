"""An ensemble keeps the staging records of one lattice between calls: they count as its device
memory, and they give way where the budget has room for a lattice but not for them too."""
from __future__ import annotations

import numpy as np
import pytest

import misa_b200 as mb
from scenarios import A0, MASS, make

pytestmark = pytest.mark.gpu
CELLS = (24, 22, 20)


def _ensemble(sc, budget=0):
    return mb.Ensemble(sc.tables, lattice_const=A0, mass=MASS, dt=1.0, cutoff=sc.cutoff, stencil_skin=sc.skin,
                       hbm_budget_bytes=budget)


def test_kept_records_are_counted_and_given_back():
    import torch
    sc = make(cells=CELLS, seed=141)
    lattice, records = mb.Ensemble.lattice_bytes(CELLS), 104 * sc.box.shape[0]
    with _ensemble(sc) as ens:
        base = ens.info()["device_bytes"]
        free = torch.cuda.mem_get_info()[0]
        slots = [ens.add(CELLS, sc.box) for _ in range(3)]
        used = free - torch.cuda.mem_get_info()[0]
        ens.run(1)
        for s in slots:
            ens.download(s)
            ens.remove(s)
        kept = ens.info()["device_bytes"] - base
        # three lattices and one set of records, to the allocator's 2 MiB granule each
        assert 3 * lattice + records <= used <= 3 * lattice + records + 4 * (2 << 20)
        assert kept >= records


@pytest.mark.parametrize("room", [0, 1])
def test_kept_records_give_way_to_lattices(room):
    # room for two lattices, and for the records as well while there is one lattice, or not
    sc = make(cells=CELLS, seed=142)
    lattice, records = mb.Ensemble.lattice_bytes(CELLS), 104 * sc.box.shape[0]
    with _ensemble(sc) as ens:
        base = ens.info()["device_bytes"]
        ens.add(CELLS, sc.box)
        ens.add(CELLS, sc.box)
        arrays = ens.info()["device_bytes"] - base - 2 * lattice - records
    budget = base + arrays + 2 * lattice + room * (records - 1)
    with _ensemble(sc, budget) as ens:
        first = ens.add(CELLS, sc.box)
        assert ens.info()["device_bytes"] <= budget
        ens.run(1)
        second = ens.add(CELLS, sc.box)
        with pytest.raises(mb.MbError, match="budget"):
            ens.add(CELLS, sc.box)
        assert ens.info()["device_bytes"] <= budget
        ens.run(2)
        a, b = ens.download(first)[0], ens.download(second)[0]
        assert ens.info()["device_bytes"] <= budget
    assert np.array_equal(a["id"], b["id"]) and np.isfinite(a["x"]).all() and np.isfinite(b["x"]).all()

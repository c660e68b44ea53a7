"""Small records through the shared host copies: once a large lattice has brought the slots in,
copies of fewer chunks than slots (2 to 8 MiB), of more, and with a short last chunk go through
them in the same ensemble."""
from __future__ import annotations

import numpy as np
import pytest

import misa_b200 as mb
from scenarios import A0, MASS, make

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def test_small_copies_after_a_large_one():
    cells = [(22, 22, 22), (24, 25, 23), (32, 32, 32), (33, 34, 35), (41, 42, 43), (22, 22, 22)]
    scs = [make(cells=c, vacancy=0.01, seed=161 + k) for k, c in enumerate(cells)]
    big = make(cells=(56, 57, 55), vacancy=0.01, seed=160)
    sizes = [104 * sc.box.shape[0] / MIB for sc in scs]
    assert 2 < min(sizes) < 3 and sum(s < 8 for s in sizes) >= 4 and 14 < max(sizes) < 16
    assert all(104 * sc.box.shape[0] % MIB for sc in scs) and 104 * big.box.shape[0] >= 32 * MIB
    with mb.Ensemble(big.tables, lattice_const=A0, mass=MASS, dt=1.0, cutoff=big.cutoff, stencil_skin=big.skin) as ens:
        for _ in range(2):  # 70 MiB up: the slots are taken
            ens.remove(ens.add(big.cells, big.box))
        slots = [ens.add(sc.cells, sc.box) for sc in scs]
        got = [ens.download(s)[0] for s in slots]
    for sc, box in zip(scs, got):
        live = sc.box["type"] >= 0
        assert np.array_equal(box["id"], sc.box["id"]) and np.array_equal(box["type"], sc.box["type"])
        for k in ("x", "v"):  # positions are kept as displacements: one rounding each way
            assert np.max(np.abs(box[k][live] - sc.box[k][live])) <= 4e-14, k

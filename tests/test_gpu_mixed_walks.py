"""One mixed-precision lattice walks by bricks or by linear items, whichever keeps the GPU
busier; in a batch it always walks linear items.  Alone and in a batch must give bitwise the
same positions and forces: a size whose bricks pay, and ragged ones whose do not."""
from __future__ import annotations

import numpy as np
import pytest

import misa_b200 as mb
from scenarios import A0, MASS, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(96, 96, 96), (32, 16, 9), (33, 20, 7), (65, 9, 12)])
def test_a_lattice_walks_alike_alone_and_in_a_batch(cells):
    sc = make(cells=cells, temperature=600.0, vacancy=0.005, seed=71, jitter=0.05)
    other = make(cells=(6, 7, 8), seed=72)
    kw = dict(lattice_const=A0, mass=MASS, dt=1.0, cutoff=sc.cutoff, stencil_skin=sc.skin)
    with mb.Sim(sc.cells, sc.tables, precision=mb.MB_PREC_MIXED, **kw) as sim:
        sim.upload(sc.box)
        sim.run(2)
        alone = sim.download()[0]
    with mb.Ensemble(sc.tables, **kw) as ens:
        slot = ens.add(sc.cells, sc.box)
        ens.add(other.cells, other.box)
        ens.run(2)
        batched = ens.download(slot)[0]
    for k in ("x", "v", "f", "rho", "df"):
        assert np.array_equal(alone[k], batched[k]), k

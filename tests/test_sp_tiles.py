"""Tiles of the sample-packed colour pass whose width is no power of two: even
and odd numbers of temperatures, a last tile that is partly filled, several
sample words.  Words and counts equal the oracle's after two sweeps; tolerance
0."""
import os

import numpy as np
import pytest

from conftest import ROOT
from test_sp import SEEDS, OracleSP, eagb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,Lz,bc,nb,NR,nw,tile", [
    (12, 48, eagb.EA_OBC, 24, 4, 2, 0),   # the width the size rule takes
    (10, 41, eagb.EA_PBC, 23, 4, 3, 0),   # odd Lz: three colours; one word a lane
    (6, 10, eagb.EA_OBC, 24, 4, 3, 11),
    (6, 10, eagb.EA_PBC, 13, 3, 2, 7),    # 273 triples a tile
    (4, 4, eagb.EA_OBC, 64, 1, 2, 3),
    (4, 4, eagb.EA_OBC, 2, 1, 2, 64),     # a tile wider than the colour
])
def test_tile_widths(L, Lz, bc, nb, NR, nw, tile):
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N32.npz"))
    k = np.round(np.linspace(0, 31, nb)).astype(int)
    betas, cum = d["betas"][k], np.ascontiguousarray(d["cum"][k])
    job = eagb.SpJob(L, Lz, betas, cum, nrep=NR, nwords=nw, bc=bc, seeds=SEEDS, jobid=4)
    job.cum = cum
    if tile:
        job.set_tile(tile)
    orc = OracleSP(job, 4)
    job.sweeps(2)
    orc.sweeps(2)
    assert np.array_equal(job.get_spins(), orc.S)
    assert np.array_equal(job.energy(), orc.energy())
    job.close()

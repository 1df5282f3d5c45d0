"""Energy count, tempering and permute of the sample-packed layout at the edges
of their forms: one and two words a lane (odd and even NB), rows of whole and
of partial 32-byte sectors, several column slices and one, more lane groups
than a tile has sites, tiles with a remainder, equal temperatures, the fewest
and the most temperatures.  Counts, energies, slot ids, acceptances, masks and
words equal the oracle's; tolerance 0."""
import os

import numpy as np
import pytest

from conftest import ROOT
from test_sp import SEEDS, OracleSP, eagb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,Lz,bc,nb,NR,nw", [
    (3, 3, eagb.EA_PBC, 2, 1, 1),      # two slots, one replica
    (2, 3, eagb.EA_OBC, 4, 1, 2),      # 128 groups for 12 sites
    (4, 6, eagb.EA_OBC, 64, 10, 1),    # 320 lanes: two column slices; temperatures twice each
    (5, 5, eagb.EA_PBC, 33, 3, 1),     # one word a lane, rows of 264 bytes
    (4, 4, eagb.EA_PBC, 61, 9, 1),     # one word a lane, three slices
    (8, 9, eagb.EA_OBC, 20, 2, 3),     # rows of 160 bytes, odd Lz
    (6, 10, eagb.EA_PBC, 22, 4, 2),    # even rows of 176 bytes
    (12, 24, eagb.EA_OBC, 24, 4, 2),   # production columns, tiles with a remainder
    (16, 32, eagb.EA_PBC, 8, 2, 1),    # 32 groups: the tile is the widest the counters take
])
def test_count_tempering_permute(L, Lz, bc, nb, NR, nw):
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N32.npz"))
    k = np.round(np.linspace(0, 31, nb)).astype(int)
    betas, cum = d["betas"][k], np.ascontiguousarray(d["cum"][k])
    job = eagb.SpJob(L, Lz, betas, cum, nrep=NR, nwords=nw, bc=bc, seeds=SEEDS, jobid=3)
    job.cum = cum
    orc = OracleSP(job, 3)
    for _ in range(2):
        job.sweeps(1)
        orc.sweeps(1)
        assert np.array_equal(job.energy(), orc.energy())
        job.parallel_tempering()
        E, M = orc.pt()
        gE, gperm, gacc, gM = job.tempering()
        assert np.array_equal(gE, E) and np.array_equal(gM, M)
        assert np.array_equal(gperm, orc.perm) and np.array_equal(gacc, orc.acc)
        assert np.array_equal(job.get_spins(), orc.S)
    job.close()

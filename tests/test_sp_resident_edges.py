"""The resident bin kernel at the edges of its split: CTAs with no or one site
of a colour, one and three colours' worth of barriers, fewest and most
temperatures (counts kept CTA by CTA and added up by atomics), equal
temperatures, more units than one wave of clusters, columns of more sites than
a warp.  Averages, words, tempering state and counters equal the oracle's over
two bins; tolerance 0."""
import os

import numpy as np
import pytest

from conftest import ROOT
from test_sp import SEEDS, OracleSP, eagb, oracle_bin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,Lz,bc,nb,NR,nw,cad", [
    (2, 3, eagb.EA_OBC, 2, 1, 1, (3, 1, 1, 1)),     # 12 sites: a site a CTA
    (3, 3, eagb.EA_PBC, 5, 2, 1, (2, 2, 1, 2)),     # three colours, 27 sites
    (4, 6, eagb.EA_OBC, 64, 1, 1, (2, 1, 2, 1)),   # counts by atomics; temperatures twice each
    (3, 5, eagb.EA_PBC, 63, 2, 1, (2, 1, 1, 1)),    # the same, counted in a phase of its own
    (4, 4, eagb.EA_PBC, 33, 3, 2, (2, 1, 1, 3)),    # more slots than warps
    (4, 8, eagb.EA_OBC, 8, 10, 16, (1, 2, 1, 1)),   # 160 units
    (10, 50, eagb.EA_OBC, 6, 4, 2, (1, 2, 2, 1)),   # 157 sites of a colour a CTA and slot
])
def test_resident_edges(L, Lz, bc, nb, NR, nw, cad):
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N32.npz"))
    k = np.round(np.linspace(0, 31, nb)).astype(int)
    betas, cum = d["betas"][k], np.ascontiguousarray(d["cum"][k])
    job = eagb.SpJob(L, Lz, betas, cum, nrep=NR, nwords=nw, bc=bc, seeds=SEEDS, jobid=5)
    job.cum = cum
    job.set_bin_kernel(eagb.EA_BIN_RESIDENT)
    orc = OracleSP(job, 5)
    for _ in range(2):
        got = job.run_bin(*cad, cluster=False)
        assert np.array_equal(got, oracle_bin(orc, *cad, False))
    E, perm, acc, M = job.tempering()
    assert np.array_equal(job.get_spins(), orc.S)
    assert np.array_equal(perm, orc.perm) and np.array_equal(acc, orc.acc)
    assert job.counter() == (orc.it, orc.step)
    U2 = job.energy()
    assert np.array_equal(U2, orc.energy())
    job.close()

"""Per-item colour pass at the edges of its rounds and queues: fewer items than
a warp, items that do not fill the last round, one and several sample words,
temperatures at which nearly no and nearly every half of a random word is
needed (all of them cold, all of them hot, both), odd and large numbers of
columns, three colours.  Words equal the oracle's; tolerance 0."""
import os

import numpy as np
import pytest

from conftest import ROOT
from test_sp import SEEDS, OracleSP, eagb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,Lz,bc,rows,NR,nw", [
    (2, 2, eagb.EA_PBC, [0, 31], 1, 1),                     # 8 items a colour
    (3, 3, eagb.EA_OBC, [0, 1, 2], 3, 1),                   # cold; three colours
    (4, 8, eagb.EA_PBC, [28, 29, 30, 31], 2, 2),            # hot
    (5, 9, eagb.EA_OBC, list(range(0, 32, 3)), 5, 1),       # 11 temperatures
    (8, 16, eagb.EA_OBC, [0, 8, 16, 24, 31], 7, 3),
    (6, 12, eagb.EA_PBC, sorted(list(range(32)) * 2), 4, 1),  # 64 temperatures, 256 columns
    (12, 50, eagb.EA_OBC, list(range(0, 32, 2)), 4, 1),     # more than one round a thread
])
def test_pass_matches_oracle(L, Lz, bc, rows, NR, nw):
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N32.npz"))
    betas, cum = d["betas"][rows], np.ascontiguousarray(d["cum"][rows])
    job = eagb.SpJob(L, Lz, betas, cum, nrep=NR, nwords=nw, bc=bc, seeds=SEEDS, jobid=3)
    job.cum = cum
    job.set_tile(0)
    orc = OracleSP(job, 3)
    for _ in range(3):
        job.sweeps(1)
        orc.sweeps(1)
        assert np.array_equal(job.get_spins(), orc.S)
    job.close()

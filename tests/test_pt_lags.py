"""Tempering draws from generators in any position: the word that a draw is
xored with may lie ahead of the one it writes, beside it or behind it.  One
bin of each against the oracle; tolerance 0."""
import numpy as np
import pytest

import oracle_py as O
from test_batch import MASTERS, eagb, lut

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d1,d2,d3", [(-24, -55, -61), (-24, -55, 5), (-24, -55, 31), (-24, -55, 1), (-24, -55, 0),
                                      (3, -55, 2), (-1, 7, 9), (-40, -33, 32)])
def test_lags(d1, d2, d3):
    betas, cum = lut("T06_16_N32")
    job = eagb.new_job(8, 8, betas, cum, nsamples=2, bc=O.PBC, masters=MASTERS, iter0=0, jobid=4)
    sim = O.Sim(8, 8, betas, cum, nbits=2, bc=O.PBC, masters=MASTERS, itmax=2)
    gen, pt = job.get_generators()
    for states in (pt, sim.pt):
        for h in states:
            h.ip1, h.ip2, h.ip3 = ((h.ip + d) & 255 for d in (d1, d2, d3))
    job.set_generators(gen, pt)
    avg, hist = job.run_bin(2, 2, 1, 1, cluster=False)
    sim.run_bin(2, 2, 1, 1, iter0=0, jobid=4, cluster=False)
    assert np.array_equal(avg, sim.avgE) and np.array_equal(hist, sim.hist)
    assert np.array_equal(job.get_permutations()[0], sim.wctb)
    assert O.as_bytes(job.get_generators()[1]) == O.as_bytes(sim.pt)
    job.close()

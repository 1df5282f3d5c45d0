"""Multispin cluster moves at the edges of their forms: lattices moved whole in
one CTA (smallest, largest, one and several chunks of planes), in slabs (equal
heights and a shorter last one, thin slabs of wide planes), and with planes
beyond shared memory; the z wrap, and site 0's bond test where L is not a power
of two, under both cluster rules.  Two bins with moves equal the oracle's, alone
and in a batch; tolerance 0."""
import importlib.util
import os

import numpy as np
import pytest

import oracle_py as O
from conftest import ROOT

spec = importlib.util.spec_from_file_location("eagb", os.path.join(ROOT, "ea-lcd-mc_gb300", "eagb.py"))
eagb = importlib.util.module_from_spec(spec)
spec.loader.exec_module(eagb)

MASTERS = (0x1234567890ABCDEF, 0x0FEDCBA987654321, 0x1111222233334444, 0x5555666677778888)
pytestmark = pytest.mark.gpu


def lut(nb):
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N32.npz"))
    k = np.round(np.linspace(0, 31, nb)).astype(int)
    return d["betas"][k], d["cum"][k]


def check(job, sim, ns):
    for s in range(ns):
        ev, od = job.get_spins(s)
        assert np.array_equal(ev, sim.spins[s, 0]) and np.array_equal(od, sim.spins[s, 1])


@pytest.mark.parametrize("L,Lz,bc,nb,ns,exact", [
    (8, 8, O.PBC, 4, 3, False),
    (8, 32, O.OBC, 3, 2, False),       # two chunks of 16 planes
    (16, 256, O.PBC, 2, 1, False),     # 65536 sites: the largest moved whole
    (24, 112, O.PBC, 2, 1, False),     # whole, L not a power of two
    (24, 112, O.OBC, 2, 1, True),
    (24, 120, O.PBC, 2, 1, False),     # slabs of 40 planes, the z wrap between the first and the last
    (24, 136, O.OBC, 2, 1, True),      # slabs of 46, 46 and 44
    (64, 24, O.PBC, 2, 1, False),      # wide planes: two slabs of 12
    (88, 8, O.OBC, 2, 1, False),
    (96, 8, O.PBC, 2, 1, False),       # planes beyond shared memory
])
def test_moves_match_oracle(L, Lz, bc, nb, ns, exact):
    betas, cum = lut(nb)
    job = eagb.new_job(L, Lz, betas, cum, nsamples=ns, NR=4, bc=bc, masters=MASTERS, iter0=0, jobid=2)
    if exact:
        eagb._ck(eagb.lib().ea_set_cluster_rule(job.ctx, 1))
    sim = O.Sim(L, Lz, betas, cum, nbits=ns, NR=4, bc=bc, masters=MASTERS, itmax=1)
    it = 0
    for _ in range(2):
        avg, _ = job.run_bin(itmax=1, houfr=1, mesfr=1, ptfr=1, cluster=True)
        it = sim.run_bin(itmax=1, houfr=1, mesfr=1, ptfr=1, iter0=it, jobid=2, cluster_exact=exact)
        assert np.array_equal(avg, sim.avgE)
    check(job, sim, ns)
    job.close()


def test_batch_of_all_forms():
    """Jobs moved whole, in slabs and in global memory in one batch."""
    shapes = [(8, 8, O.PBC, 4, 3), (24, 120, O.PBC, 2, 1), (96, 8, O.PBC, 2, 1), (16, 40, O.OBC, 3, 2)]
    jobs, sims = [], []
    for k, (L, Lz, bc, nb, ns) in enumerate(shapes):
        betas, cum = lut(nb)
        jobs.append(eagb.new_job(L, Lz, betas, cum, nsamples=ns, NR=4, bc=bc, masters=MASTERS, iter0=0, jobid=k))
        sims.append(O.Sim(L, Lz, betas, cum, nbits=ns, NR=4, bc=bc, masters=MASTERS, itmax=2))
    batch = eagb.Batch(jobs)
    its = [0] * len(jobs)
    for _ in range(2):
        batch.run_bin(itmax=2, houfr=2, mesfr=1, ptfr=1, cluster=True)
        for k, sim in enumerate(sims):
            its[k] = sim.run_bin(itmax=2, houfr=2, mesfr=1, ptfr=1, iter0=its[k], jobid=k)
            assert np.array_equal(jobs[k].bin_results()[0], sim.avgE)
    batch.sync()
    for job, sim, sh in zip(jobs, sims, shapes):
        check(job, sim, sh[4])
    batch.close()
    for job in jobs:
        job.close()

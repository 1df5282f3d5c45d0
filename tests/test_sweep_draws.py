"""Random words of the multispin half-sweep at the edges of their forms: the
temperature counts where the pre-search tables change their bits, the shortest
and the longest ladder, thresholds that leave every, some and no half of the
second and third word to be drawn, every tile width, and a batch whose jobs'
tables have different bits.  Equal to the oracle's sweeps; tolerance 0."""
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


def lut(nb, kind):
    """ladder: the golden one stretched over nb; dense: every byte equally
    likely; never: byte 0 always; mixed: the three in turn."""
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N32.npz"))
    k = np.round(np.linspace(0, 31, nb)).astype(int)
    betas, cum = d["betas"][k], d["cum"][k].copy()
    full = np.uint64(0xFFFFFFFFFFFFFFFF)
    dense = np.append(np.arange(1, 256, dtype=np.uint64) << np.uint64(56), full)
    for b in range(nb):
        if kind == "dense" or kind == "mixed" and b % 3 == 1:
            cum[b] = dense[:cum.shape[1]]
        elif kind == "never" or kind == "mixed" and b % 3 == 2:
            cum[b] = full
    return betas, cum


def check(job, sim, ns):
    for s in range(ns):
        ev, od = job.get_spins(s)
        assert np.array_equal(ev, sim.spins[s, 0]) and np.array_equal(od, sim.spins[s, 1])


@pytest.mark.parametrize("nb,NR,ns,kind", [
    (2, 8, 1, "ladder"), (2, 2, 3, "dense"),
    (40, 8, 1, "ladder"), (41, 8, 1, "mixed"),
    (72, 4, 1, "mixed"), (73, 4, 1, "ladder"),
    (128, 2, 1, "mixed"), (129, 2, 1, "dense"),
    (255, 8, 1, "mixed"), (12, 8, 2, "never"),
])
def test_sweeps_match_oracle(nb, NR, ns, kind, monkeypatch):
    betas, cum = lut(nb, kind)
    sim = O.Sim(8, 8, betas, cum, nbits=ns, NR=NR, bc=O.PBC, masters=MASTERS, itmax=1)
    sim.run_bin(itmax=1, houfr=1, mesfr=1, ptfr=2, iter0=0, jobid=3, cluster=False)
    for kt in {8: (1, 2, 4), 4: (2, 4, 8), 2: (4, 8, 16)}[NR]:  # a width that does not fit is chosen by size
        monkeypatch.setenv("EAGB_KT", str(kt))
        job = eagb.new_job(8, 8, betas, cum, nsamples=ns, NR=NR, bc=O.PBC, masters=MASTERS, iter0=0, jobid=3)
        avg, _ = job.run_bin(itmax=1, houfr=1, mesfr=1, ptfr=2, cluster=False)
        assert np.array_equal(avg, sim.avgE)
        check(job, sim, ns)
        job.close()


def test_batch_of_table_sizes():
    nbs = (3, 40, 41, 73, 130)
    jobs, sims = [], []
    for k, nb in enumerate(nbs):
        betas, cum = lut(nb, "mixed")
        jobs.append(eagb.new_job(8, 8, betas, cum, nsamples=1, NR=4, bc=O.OBC, masters=MASTERS, iter0=0, jobid=k))
        sims.append(O.Sim(8, 8, betas, cum, nbits=1, NR=4, bc=O.OBC, masters=MASTERS, itmax=1))
    batch = eagb.Batch(jobs)
    batch.run_bin(itmax=1, houfr=1, mesfr=1, ptfr=2, cluster=False)
    batch.sync()
    for k, sim in enumerate(sims):
        sim.run_bin(itmax=1, houfr=1, mesfr=1, ptfr=2, iter0=0, jobid=k, cluster=False)
        check(jobs[k], sim, 1)

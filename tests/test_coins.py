"""Cluster coins (the bits [U < 0.5] of the reference's cuRAND doubles, drawn
without the doubles) at the edges of their split: streams in one segment and
in several, moves that end inside a row of the 4096 streams, and sequences
started at an offset (below, at and above whole rows; odd).  The job's words
after several moves equal the oracle's, which draws the doubles with the host
cuRAND generator; tolerance 0."""
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


# L, Lz, NB (rows of the 32-temperature set), samples, offset of the sequence
@pytest.mark.parametrize("L,Lz,nb,ns,offset", [
    (8, 8, 5, 1, 0),            # 5120 coins a move: one row and a quarter
    (8, 8, 3, 1, 4095),         # below one row; the last stream alone is ahead
    (8, 8, 32, 31, 1000003),    # 248 rows: the largest of one segment; coins off a word boundary
    (8, 16, 32, 16, 0),         # 256 rows: the smallest of two segments
    (8, 16, 32, 17, 4097),      # two segments, one draw into a row
    (24, 16, 32, 5, 12289),     # 720 rows: five segments, L not a power of two
])
def test_coins_match_curand(L, Lz, nb, ns, offset):
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N32.npz"))
    k = np.round(np.linspace(0, 31, nb)).astype(int)
    betas, cum = d["betas"][k], d["cum"][k]
    job = eagb.new_job(L, Lz, betas, cum, nsamples=ns, NR=4, bc=O.OBC, masters=MASTERS, iter0=0, jobid=2)
    sim = O.Sim(L, Lz, betas, cum, nbits=ns, NR=4, bc=O.OBC, masters=MASTERS, itmax=2)
    gen, pt = job.get_generators()
    gen.cuda_rng_offset = offset
    job.set_generators(gen, pt)
    sim.cuda_rng_offset = offset
    it = 0
    for _ in range(2):
        avg, _ = job.run_bin(itmax=2, houfr=1, mesfr=1, ptfr=1, cluster=True)
        it = sim.run_bin(itmax=2, houfr=1, mesfr=1, ptfr=1, iter0=it, jobid=2)
        assert np.array_equal(avg, sim.avgE)
    for s in range(ns):
        ev, od = job.get_spins(s)
        assert np.array_equal(ev, sim.spins[s, 0]) and np.array_equal(od, sim.spins[s, 1])
    gen, _ = job.get_generators()
    assert gen.cuda_rng_offset == sim.cuda_rng_offset
    job.close()

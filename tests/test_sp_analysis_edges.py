"""Plane counts and correlations at the edges of their launches: few and many
slots a block, planes smaller than the lane groups and large ones, one and
several words and pairs, distances that do not fill a block, both boundary
conditions, overlaps that vanish (sign 0).  Counts equal those made from the
spin words, correlations the restatement in Python floats; tolerance 0."""
import os

import numpy as np
import pytest

from conftest import ROOT
from test_analysis import SEEDS, eagb, restated_correlations

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,Lz,bc,nb,NR,nrep,nw,dmax", [
    (2, 2, eagb.EA_PBC, 2, 2, 2, 1, 1),      # 128 groups for 4 sites; vanishing overlaps
    (2, 3, eagb.EA_OBC, 64, 2, 2, 1, 2),     # 64 slots
    (17, 4, eagb.EA_OBC, 3, 5, 4, 2, 3),     # odd planes, two pairs of five replicas, two words
    (4, 11, eagb.EA_PBC, 5, 6, 6, 1, 8),     # nine distances: the second group has one
    (20, 3, eagb.EA_PBC, 61, 2, 2, 1, 0),    # 4 groups of 100 sites; distance 0 alone
])
def test_counts_and_correlations(L, Lz, bc, nb, NR, nrep, nw, dmax):
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N32.npz"))
    k = np.round(np.linspace(0, 31, nb)).astype(int)
    job = eagb.SpJob(L, Lz, d["betas"][k], d["cum"][k], nrep=NR, nwords=nw, bc=bc, seeds=SEEDS)
    S = np.random.default_rng(L * 100 + Lz).integers(0, 1 << 64, (nw, L * L * Lz, NR, nb), np.uint64)
    job.set_spins(S)
    diff = job.plane_overlaps(nrep)
    want = np.zeros_like(diff)
    for p in range(nrep // 2):
        x = S[:, :, 2 * p, :] ^ S[:, :, 2 * p + 1, :]
        bits = (x[..., None] >> np.arange(64, dtype=np.uint64)) & np.uint64(1)
        want[:, :, p] = np.transpose(bits.reshape(nw, Lz, L * L, nb, 64).sum(2), (0, 3, 2, 1))
    assert np.array_equal(diff, want)
    assert np.array_equal(job.plane_correlations(nrep, dmax), restated_correlations(diff, L * L, Lz, bc == eagb.EA_PBC, dmax))
    job.close()

"""Cluster labelling by runs at the edges of its forms: 8, 4, 2 and 1 samples at
a time in shared memory, flat lattices beyond them, slabs of a tall tube (8, 4
and 1 samples), columns of one and several chunks of planes with a shorter
last one, the z wrap, the corner bond of odd open tubes.  One move on states
with small and with percolating clusters equals the oracle's; tolerance 0."""
import importlib.util
import os

import numpy as np
import pytest

import oracle_py as O
from conftest import ROOT

spec = importlib.util.spec_from_file_location("eagb", os.path.join(ROOT, "ea-lcd-mc_gb300", "eagb.py"))
eagb = importlib.util.module_from_spec(spec)
spec.loader.exec_module(eagb)

pytestmark = pytest.mark.gpu
SEEDS = (0x1234567890ABCDEF, 0x0FEDCBA987654321, 0x1111222233334444, 0x5555666677778888)


@pytest.mark.parametrize("L,Lz,bc", [
    (2, 2, O.PBC), (3, 3, O.OBC), (5, 31, O.OBC), (5, 32, O.PBC), (4, 63, O.OBC), (3, 95, O.PBC),
    (16, 40, O.OBC),     # the tallest at 8 samples
    (16, 42, O.PBC),     # 4 samples
    (16, 80, O.OBC),     # 2 samples
    (16, 128, O.PBC),    # 2 samples, the largest lattice labelled whole
    (17, 112, O.OBC),    # odd, 32368 sites
    (80, 5, O.PBC),      # 1 sample
    (128, 2, O.OBC),     # wide planes: one thread a site
    (20, 96, O.PBC),     # slabs, 8 samples
    (21, 75, O.OBC),     # slabs of an odd open tube: the corner bond joins the first and last
    (46, 18, O.PBC),     # slabs, 4 samples
    (65, 9, O.OBC),      # slabs, 1 sample
])
def test_move_matches_oracle(L, Lz, bc):
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N6.npz"))
    nb, NR, nw, nc = 3, 2, 1 + (L <= 5), 2
    betas, cum = d["betas"][:nb], d["cum"][:nb]
    job = eagb.SpJob(L, Lz, betas, cum, nrep=NR, nwords=nw, bc=bc, seeds=SEEDS)
    V = L * L * Lz
    rng = np.random.default_rng(L * 1000 + Lz)
    S = rng.integers(0, 1 << 64, (nw, V, NR, nb), np.uint64)
    noise = rng.integers(0, 1 << 64, (3, nw, V), np.uint64)
    S[:, :, 1, 0] = S[:, :, 0, 0] ^ (noise[0] & noise[1])   # slot 0: a quarter of the spins differ; slot 1: half
    job.set_spins(S)
    nbr = eagb.sp_graph(L, Lz, bc)[0]
    key = SEEDS[3] ^ 0xC2B2AE3585EBCA6B
    ref = S.copy()
    # two replicas are one group, in either order
    job.houdayer(nc)
    got = job.get_spins()
    oks = []
    for r1, r2 in ((0, 1), (1, 0)):
        x = ref.copy()
        O.sp_cluster(V, NR, nb, nw, nbr, nc, 0, r1, r2, 1, key, x)
        oks.append(np.array_equal(x, got))
    assert any(oks)
    assert not np.array_equal(got, S)
    job.close()

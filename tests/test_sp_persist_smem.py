"""The persistent bin kernel beside the most shared memory a move takes: 32,768
sites in two wide planes, 224 KB, the largest lattice labelled on chip.  Words
and tempering state equal the graph's and the oracle's; tolerance 0."""
import numpy as np
import pytest

from test_sp import OracleSP, eagb, new_job, oracle_bin

pytestmark = pytest.mark.gpu


def test_moves_of_the_largest_lattice_on_chip():
    cad = (1, 1, 1, 1)
    a, b = (new_job(128, 2, eagb.EA_PBC, "T08_16_N4", 2, 1, jobid=5) for _ in range(2))
    a.set_bin_kernel(eagb.EA_BIN_GRAPH)
    b.set_bin_kernel(eagb.EA_BIN_PERSISTENT)
    orc = OracleSP(a, 5)
    va, vb = (j.run_bin(*cad, cluster=True) for j in (a, b))
    want = oracle_bin(orc, *cad, True)
    assert np.array_equal(va, want) and np.array_equal(vb, want)
    assert np.array_equal(a.get_spins(), orc.S) and np.array_equal(b.get_spins(), orc.S)
    assert all(np.array_equal(x, y) for x, y in zip(a.tempering(), b.tempering()))
    a.close()
    b.close()


@pytest.mark.parametrize("L,Lz,nb,NR,nw,tile", [
    (12, 48, 53, 12, 2, None),   # the default tile: 8 sites, 231,728 bytes
    (6, 8, 61, 6, 2, 12),        # the widest that fits: 231,648 bytes
])
def test_the_widest_tiles(L, Lz, nb, NR, nw, tile):
    import os
    from conftest import ROOT
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N32.npz"))
    k = np.round(np.linspace(0, 31, nb)).astype(int)
    a, b = (eagb.SpJob(L, Lz, d["betas"][k], np.ascontiguousarray(d["cum"][k]), nrep=NR, nwords=nw, bc=eagb.EA_OBC)
            for _ in range(2))
    a.set_bin_kernel(eagb.EA_BIN_GRAPH)
    b.set_bin_kernel(eagb.EA_BIN_PERSISTENT)
    if tile:
        b.set_tile(tile)
    for cluster in (False, True):
        assert np.array_equal(*(j.run_bin(1, 1, 1, 1, cluster=cluster) for j in (a, b)))
    assert np.array_equal(a.get_spins(), b.get_spins())
    a.close()
    b.close()

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

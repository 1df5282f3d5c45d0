"""Energy count of jobs with few (replica, slot) columns and many sample words,
whose tiles would be the widest: every form's launch stays within the shared
memory it may take (CPU, on a runtime without a GPU), and the counts equal the
oracle's (tolerance 0)."""
import ctypes as C
import os

import numpy as np
import pytest

from conftest import ROOT
from test_sp import SEEDS, OracleSP, eagb


def ladder(nb):
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N32.npz"))
    k = np.round(np.linspace(0, 31, nb)).astype(int)
    return d["betas"][k], np.ascontiguousarray(d["cum"][k])


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    import fakecuda
    return fakecuda.load(tmp_path_factory.mktemp("fake"))


# words: the fewest that once asked for too much, and more (42 sites a lane)
@pytest.mark.parametrize("L,Lz,nb,NR,nw", [
    (24, 192, 2, 1, 29), (24, 192, 2, 1, 220), (24, 192, 4, 2, 28), (12, 48, 4, 2, 437), (24, 192, 12, 1, 28),
    (24, 192, 3, 1, 160), (24, 192, 4, 1, 120), (24, 192, 11, 1, 40), (24, 192, 7, 2, 40), (24, 192, 15, 1, 40),
])
def test_every_launch_fits(fake, L, Lz, nb, NR, nw):
    eb, fk = fake
    lib = eb.lib()
    betas, cum = ladder(nb)
    g = eb.SpGeom(L, Lz, nb, NR, nw, eb.EA_OBC)
    h = C.c_void_p()
    eb._ck(lib.ea_sp_create(C.byref(g), 0, C.byref(h)))
    fk.fake_reset()
    try:
        eb._ck(lib.ea_sp_set_temperatures(h, eb.P(betas), eb.P(cum)))
        eb._ck(lib.ea_sp_energy(h, None))
        eb._ck(lib.ea_sp_parallel_tempering(h))
        cad = eb.Cadence(2, 2, 1, 1, 0, 0)
        for mode in (eb.EA_BIN_GRAPH, eb.EA_BIN_PERSISTENT):
            eb._ck(lib.ea_sp_set_bin_kernel(h, mode))
            eb._ck(lib.ea_sp_run(h, C.byref(cad), None))
        b = C.c_void_p()
        eb._ck(lib.ea_sp_batch_create((C.c_void_p * 1)(h), 1, C.byref(b)))
        try:
            for mode in (eb.EA_BIN_AUTO, eb.EA_BIN_PERSISTENT):
                eb._ck(lib.ea_sp_batch_set_bin_kernel(b, mode))
                eb._ck(lib.ea_sp_batch_run(b, C.byref(cad)))
        finally:
            lib.ea_sp_batch_destroy(b)
    finally:
        lib.ea_sp_destroy(h)
    assert fk.fake_refused() == b""


@pytest.mark.gpu
@pytest.mark.parametrize("L,Lz,bc,nb,NR,nw", [
    (24, 192, eagb.EA_OBC, 2, 1, 29),   # 144 groups: 66 KB for the sites of the widest tile
    (12, 48, eagb.EA_PBC, 4, 2, 437),   # 36 groups
])
def test_counts_of_few_columns(L, Lz, bc, nb, NR, nw):
    betas, cum = ladder(nb)
    job = eagb.SpJob(L, Lz, betas, cum, nrep=NR, nwords=nw, bc=bc, seeds=SEEDS, jobid=3)
    job.cum = cum
    orc = OracleSP(job, 3)
    want = orc.energy()
    assert np.array_equal(job.energy(), want)
    batch = eagb.SpBatch([job])
    for run, mode in ((job, eagb.EA_BIN_GRAPH), (batch, eagb.EA_BIN_AUTO), (batch, eagb.EA_BIN_PERSISTENT)):
        run.set_bin_kernel(mode)
        run.run_bin(1, 1, 1, 1, cluster=False)  # its energies are those of the words it leaves
        E = job.tempering()[0]
        orc.S = np.ascontiguousarray(job.get_spins())
        assert np.array_equal(E, 3 * job.V - orc.energy())
    batch.close()
    job.close()

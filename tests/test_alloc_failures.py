"""Allocations that fail, on a runtime without a GPU (fake_cudart.cpp): the
call that met the failure reports it, and nothing of it is left behind -- the
next calls work, with every buffer that they need."""
import ctypes as C
import os

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    import fakecuda
    return fakecuda.load(tmp_path_factory.mktemp("fake"))


def ladder(nb):
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N32.npz"))
    k = np.round(np.linspace(0, 31, nb)).astype(int)
    return d["betas"][k], np.ascontiguousarray(d["cum"][k])


def ms_job(eb, L=16, Lz=64, nb=24, NR=4, ns=2):
    job = eb.Job(eb.geom(L, Lz, nb, NR, ns, eb.EA_OBC))
    job.set_temperatures(*ladder(nb))
    return job


def sp_job(eb, L=6, Lz=24, nb=12, NR=2):
    return eb.SpJob(L, Lz, *ladder(nb), nrep=NR, bc=eb.EA_OBC)


def test_a_failure_is_reported_once(fake):
    """An allocation's error must not come back as the next launch's: that
    launch's kernel runs, so its call would fail half done."""
    eb, fk = fake
    job = ms_job(eb)
    fk.fake_fail_in(0)
    with pytest.raises(eb.EAError):
        job.houdayer()
    job.monte_carlo(1)
    job.close()
    job = sp_job(eb)
    for call in (job.houdayer, lambda: job.plane_overlaps(2), lambda: job.plane_correlations(2, 3)):
        fk.fake_fail_in(0)
        with pytest.raises(eb.EAError):
            call()
        job.sweeps(1)
    fk.fake_fail_in(0)
    with pytest.raises(eb.EAError):
        sp_job(eb)
    job.sweeps(1)
    job.close()

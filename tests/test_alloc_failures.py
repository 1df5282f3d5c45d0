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


def same_buffers(eb, fk, make, calls, last):
    """Every allocation of `calls` fails once, each on a job of its own.  The
    calls `last` then leave the buffers of a job that met no failure."""
    def held(k):
        live, bytes_ = fk.fake_live(), fk.fake_live_bytes()
        job = make()
        failed = 0
        fk.fake_fail_in(k)
        for call in calls:
            try:
                call(job)
            except eb.EAError:
                failed += 1
        fk.fake_fail_in(-1)
        for call in last:
            call(job)
        got = fk.fake_live() - live, fk.fake_live_bytes() - bytes_
        job.close()
        assert (fk.fake_live(), fk.fake_live_bytes()) == (live, bytes_)
        return got, failed

    want, failed = held(-1)
    assert not failed
    k = 0
    while True:
        got, failed = held(k)
        assert got == want, "allocation %d failed" % k
        if not failed:
            return k
        k += 1


def test_coins_of_a_move(fake):
    eb, fk = fake
    n = same_buffers(eb, fk, lambda: ms_job(eb), [lambda j: j.houdayer()], [lambda j: j.houdayer()])
    assert n >= 7   # coins, states, positions, jumps; labels, selection, overlaps
    same_buffers(eb, fk, lambda: ms_job(eb), [lambda j: j.run_bin(1, 1, 1, 1)], [lambda j: j.run_bin(1, 1, 1, 1)])


def test_buffers_that_grow(fake):
    """A growth that fails leaves no stale capacity: a smaller move or a
    shorter bin afterwards has its buffers."""
    eb, fk = fake
    for small, large in ((lambda j: j.houdayer(3), lambda j: j.houdayer(9)),
                         (lambda j: j.run_bin(2, 1, 1, 1, cluster=False), lambda j: j.run_bin(5, 1, 1, 1, cluster=False))):
        def grown(make):
            job = make()
            small(job)
            return job
        for make in (lambda: ms_job(eb), lambda: sp_job(eb), lambda: sp_job(eb, 33, 33, 6)):
            k = 0
            while True:
                live, bytes_ = fk.fake_live(), fk.fake_live_bytes()
                job = grown(make)
                want = fk.fake_live() - live, fk.fake_live_bytes() - bytes_
                fk.fake_fail_in(k)
                try:
                    large(job)
                    failed = False
                except eb.EAError:
                    failed = True
                fk.fake_fail_in(-1)
                small(job)
                got = fk.fake_live() - live, fk.fake_live_bytes() - bytes_
                job.close()
                if not failed:
                    break
                assert got == want, "allocation %d failed" % k
                k += 1


def test_temperatures_replaced(fake):
    """New temperatures whose table finds no memory: the job has none, and
    says so, until they are set again."""
    eb, fk = fake
    for job, nb, step in ((ms_job(eb), 24, lambda j: j.monte_carlo(1)), (sp_job(eb), 12, lambda j: j.sweeps(1))):
        betas, cum = ladder(nb)
        args = (job.ctx,) if hasattr(job, "ctx") else (job.h,)
        call = eb.lib().ea_set_temperatures if hasattr(job, "ctx") else eb.lib().ea_sp_set_temperatures
        fk.fake_fail_in(0)
        assert call(*args, eb.P(betas), eb.P(cum)) != 0
        with pytest.raises(eb.EAError, match="temperatures not set"):
            step(job)
        eb._ck(call(*args, eb.P(betas), eb.P(cum)))
        step(job)
        job.close()


def test_buffers_of_the_persistent_kernel(fake):
    eb, fk = fake

    def make():
        job = sp_job(eb)
        job.set_bin_kernel(eb.EA_BIN_PERSISTENT)
        return job
    bin_ = lambda j: j.run_bin(1, 1, 1, 1)
    assert same_buffers(eb, fk, make, [bin_], [bin_]) >= 4
    same_buffers(eb, fk, lambda: sp_job(eb), [bin_], [bin_])   # the resident kernel's


def test_autotuner_refuses_before_it_times(fake):
    """A refusal -- no memory, or one replica, which has no moves to label for
    -- comes before the timing runs change the job's words."""
    eb, fk = fake
    for NR, fails in ((2, 2), (1, 1)):
        job = sp_job(eb, NR=NR)
        for k in range(fails):
            fk.fake_reset()
            fk.fake_fail_in(k)
            with pytest.raises(eb.EAError):
                job.autotune()
            assert fk.fake_calls(b"launch ") == 0
        fk.fake_reset()
        job.close()


@pytest.mark.parametrize("cluster", [False, True])
def test_a_bin_without_room_for_the_resident_buffers(fake, cluster):
    """The default takes the graph, which needs none of them; the resident
    kernel, when asked for by name, says that they are missing."""
    eb, fk = fake
    for k in range(3):
        for mode in (eb.EA_BIN_AUTO, eb.EA_BIN_RESIDENT):
            job = sp_job(eb)
            job.set_bin_kernel(mode)
            assert job.bin_kernel_for(3, 4, cluster=cluster) == eb.EA_BIN_RESIDENT
            fk.fake_reset()
            fk.fake_fail_in(k + int(cluster))     # after the overlap words of a move
            if mode == eb.EA_BIN_AUTO:
                job.run_bin(3, 4, cluster=cluster)
                assert fk.fake_calls(b"cudaGraphLaunch") == 3 and not fk.fake_calls(b"launch _ZN4eagb13k_sp_resident")
                job.run_bin(3, 4, cluster=cluster)
            else:
                with pytest.raises(eb.EAError, match="out of memory"):
                    job.run_bin(3, 4, cluster=cluster)
                job.run_bin(3, 4, cluster=cluster)
            assert fk.fake_calls(b"launch _ZN4eagb13k_sp_resident") > 0
            job.close()
            fk.fake_reset()


def test_a_move_without_room_for_slab_labels(fake):
    """Wide planes (100 x 100) and a long tube: the scratch that every large
    lattice has is enough for a move."""
    eb, fk = fake
    for L, Lz in ((100, 4), (24, 60)):
        for k in (2, 3):   # overlap words, scratch; slab labels, their coins
            job = sp_job(eb, L, Lz, 4)
            fk.fake_reset()
            fk.fake_fail_in(k)
            job.houdayer(2)
            assert fk.fake_calls(b"launch _ZN4eagb12k_sp_cluster") == 1
            assert fk.fake_calls(b"launch _ZN4eagb9k_sp_slab") == 0
            fk.fake_fail_in(-1)
            job.houdayer(4)    # a larger move asks again
            assert fk.fake_calls(b"launch _ZN4eagb9k_sp_slab") > 0
            job.close()
            fk.fake_reset()

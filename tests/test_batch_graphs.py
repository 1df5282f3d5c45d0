"""Graphs of a batch's tempering cycles: how many are instantiated (CPU, on a
runtime without a GPU), and that bins that go in several pieces equal those of
the jobs alone (tolerance 0)."""
import numpy as np
import pytest

from test_alloc_failures import fake, ms_job  # noqa: F401
from test_batch import assert_same, eagb, make_jobs


@pytest.mark.parametrize("houfr,ptfr,graphs", [
    (10, 1, 1), (32, 1, 1), (40, 1, 1), (33, 1, 2), (64, 1, 1), (100, 1, 1), (101, 1, 2),   # 32 cycles at most
    (40, 0, 1), (10, 10, 1), (7, 30, 2), (3, 500, 1)])                                      # and 128 launches
def test_a_piece_is_captured_once(fake, houfr, ptfr, graphs):  # noqa: F811
    eb, fk = fake
    jobs = [ms_job(eb), ms_job(eb, 8, 16, 6)]
    batch = eb.Batch(jobs, tile=4)
    fk.fake_reset()
    for _ in range(2):
        batch.run_bin(3, houfr, 2, ptfr)
    assert fk.fake_calls(b"cudaGraphInstantiate") == graphs
    sweeps = fk.fake_calls(b"launch _ZN4eagb8kb_sweep") - 2 * 3   # less the energies of each iteration
    assert sweeps <= graphs * max(128, 2 * ptfr)
    # another cadence and back: the batch keeps two graphs (a shorter cadence may be a piece of the other)
    if graphs == 1:
        for h in (5, houfr, 5, houfr):
            batch.run_bin(1, h, 1, ptfr)
        assert fk.fake_calls(b"cudaGraphInstantiate") <= 2
    batch.close()
    for j in jobs:
        j.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cad", [(2, 33, 2, 1), (1, 40, 2, 1), (1, 5, 1, 40)])
def test_pieces_equal_jobs_alone(cad):
    alone, jobs = make_jobs()[:3], make_jobs()[:3]
    batch = eagb.Batch(jobs)
    for cluster in (True, False):
        batch.run_bin(*cad, cluster=cluster)
        batch.sync()
        for a, b in zip(alone, jobs):
            avg, hist = a.run_bin(*cad, cluster=cluster)
            got = b.bin_results()
            assert np.array_equal(avg, got[0]) and np.array_equal(hist, got[1])
            assert_same(a, b)
    batch.close()
    for j in alone + jobs:
        j.close()

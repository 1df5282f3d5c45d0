"""What a job's kernels read is uploaded on the stream they run on.  A plain
copy or fill goes through the legacy default stream, which the jobs' streams
do not wait for, and a plain copy from pageable memory may return before it
has reached the device.  CPU, on a runtime without a GPU."""

from test_alloc_failures import fake, ms_job, sp_job  # noqa: F401


def test_no_upload_beside_the_streams(fake):  # noqa: F811
    eb, fk = fake
    fk.fake_reset()
    jobs = [ms_job(eb), ms_job(eb, 8, 16, 6)]
    jobs[0].run_bin(1, 1, 1, 1)
    jobs[1].houdayer()
    batch = eb.Batch(jobs)
    batch.run_bin(1, 2, 1, 1)
    batch.close()
    sp = [sp_job(eb), sp_job(eb, 7, 21, 13)]
    for mode in (eb.EA_BIN_AUTO, eb.EA_BIN_GRAPH, eb.EA_BIN_PERSISTENT):
        sp[0].set_bin_kernel(mode)
        sp[0].run_bin(2, 4, 1, 1, cluster=True)
    for mode in (eb.EA_BIN_AUTO, eb.EA_BIN_PERSISTENT):
        batch = eb.SpBatch(sp)
        batch.set_bin_kernel(mode)
        batch.run_bin(2, 4, 1, 1, cluster=True)
        batch.close()
    sp[0].plane_correlations(2, 3)
    for j in jobs + sp:
        j.close()
    for what in (b"cudaMemcpy to device", b"cudaMemset"):
        assert fk.fake_calls(what) == 0, what

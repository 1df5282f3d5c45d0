"""Spins read back into pages that nobody has touched, at any offset in them and
beside a neighbour's data in the first and last one: the same words as into a
used array, and the neighbour's data as they were."""
import importlib.util
import mmap
import os

import numpy as np
import pytest

from conftest import ROOT

spec = importlib.util.spec_from_file_location("eagb", os.path.join(ROOT, "ea-lcd-mc_gb300", "eagb.py"))
eagb = importlib.util.module_from_spec(spec)
spec.loader.exec_module(eagb)
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 8, 4096, 65528])
def test_new_pages(offset):
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N32.npz"))
    job = eagb.new_job(16, 16, d["betas"], d["cum"], nsamples=1, NR=8, bc=eagb.EA_PBC, masters=(1, 2, 3, 4),
                       iter0=0, jobid=0)
    job.monte_carlo(2)
    ev, od = job.get_spins(0)
    size = 2 * ev.nbytes + offset + 64
    room = np.frombuffer(mmap.mmap(-1, size), np.uint8)
    if offset:
        room[offset - 8:offset] = 0xA5
    room[offset + 2 * ev.nbytes:offset + 2 * ev.nbytes + 8] = 0x5A
    out = room[offset:offset + 2 * ev.nbytes].view(np.uint64)
    eagb._ck(eagb.lib().ea_get_spins(job.ctx, 0, eagb.P(out[:ev.size]), eagb.P(out[ev.size:])))
    assert np.array_equal(out[:ev.size], ev) and np.array_equal(out[ev.size:], od)
    assert not offset or (room[offset - 8:offset] == 0xA5).all()
    assert (room[offset + 2 * ev.nbytes:offset + 2 * ev.nbytes + 8] == 0x5A).all()
    job.close()

"""Spins read back into large arrays whose pages are present in part: all of
them, the middle and the last one alone (taken for a used array), the first one
alone.  The same words each time."""
import mmap

import numpy as np
import pytest

from test_sp import eagb, new_job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("touched", [(), (0,), (0.5, -1), "all"])
def test_large_arrays(touched):
    job = new_job(12, 48, eagb.EA_OBC, "T07_16_N24", 4, 1)
    want = job.get_spins()
    assert want.nbytes >= 1 << 20
    room = np.frombuffer(mmap.mmap(-1, want.nbytes), np.uint64)
    if touched == "all":
        room[:] = 1
    else:
        for t in touched:
            room[int(t * room.size) if 0 <= t < 1 else -1] = 1
    eagb._ck(eagb.lib().ea_sp_get_spins(job.h, eagb.P(room)))
    assert np.array_equal(room, want.reshape(-1))
    job.close()

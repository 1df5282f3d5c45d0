"""Energy count of a job whose words lie beyond index 2^32 (34 GB): the words
of the last plane alone are not zero, so with couplings of zero each of its
spins leaves its two bonds along z unsatisfied and no other bond is."""
import ctypes as C

import numpy as np
import pytest

from test_sp import eagb

pytestmark = pytest.mark.gpu


def test_words_beyond_32_bits():
    import torch
    L, Lz, nb, NR = 64, 258, 64, 64
    V, G, L2 = L * L * Lz, nb * NR, L * L
    assert (V - L2) * G >= 1 << 32
    if torch.cuda.mem_get_info()[0] < 8 * V * G + (4 << 30):
        pytest.skip("needs 39 GB of GPU memory")
    lib, ck = eagb.lib(), eagb._ck
    g = eagb.SpGeom(L, Lz, nb, NR, 1, eagb.EA_PBC)
    job = C.c_void_p()
    ck(lib.ea_sp_create(C.byref(g), 0, C.byref(job)))
    try:
        words = np.random.default_rng(1).integers(0, 1 << 64, G, np.uint64)
        S = np.zeros((V, G), np.uint64)   # pages of zeros but for the last plane
        S[V - L2:] = words
        ck(lib.ea_sp_set_spins(job, eagb.P(S)))
        U2 = np.zeros((64, G), np.int32)
        ck(lib.ea_sp_energy(job, eagb.P(U2)))
    finally:
        ck(lib.ea_sp_destroy(job))
    bits = (words[None, :] >> np.arange(64, dtype=np.uint64)[:, None]) & np.uint64(1)
    assert np.array_equal(U2, (4 * L2 * bits).astype(np.int32))

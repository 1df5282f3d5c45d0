"""Plane overlaps that vanish: sign(0) = 0 for every plane size, also where
2/L^2 is not exact (14 x 14: 2/196 times 98 rounds to less than 1).  The sign
is taken from the counts; tolerance 0."""
import os

import numpy as np
import pytest

from conftest import ROOT
from test_analysis import SEEDS, analysis, eagb


def planes(L, Lz, rng, n):
    """Counts with half of the planes at exactly L^2/2."""
    diff = rng.integers(0, L * L + 1, n + (Lz,)).astype(np.int32)
    diff[..., ::2] = L * L // 2
    return diff


def sign_products(diff, L2, pbc, dmax):
    s = np.sign(L2 - 2 * diff.astype(np.int64))
    out = []
    for d in range(dmax + 1):
        a, b = (s, np.roll(s, -d, -1)) if pbc else (s[..., :s.shape[-1] - d], s[..., d:])
        p = a * b                                                   # [samples][pair][slot][z]
        out.append(p.sum((1, 3)) / (p.shape[1] * p.shape[3]))
    return np.stack(out, -1)


@pytest.mark.parametrize("L", [2, 4, 6, 14, 20, 28, 54, 56, 58])
def test_host_correlations(L):
    diff = planes(L, 6, np.random.default_rng(L), (3, 2, 2))
    for pbc in (True, False):
        C = analysis.plane_correlations(diff, L * L, pbc, 5)
        assert np.allclose(C[..., 2, 2], sign_products(diff, L * L, pbc, 5), rtol=0, atol=1e-12)
    half = np.full_like(diff, L * L // 2)
    assert not analysis.plane_correlations(half, L * L, True, 5).any()


@pytest.mark.gpu
@pytest.mark.parametrize("L", [4, 6, 14, 28])
def test_device_correlations(L):
    Lz, nb, dmax = 6, 3, 5
    d = np.load(os.path.join(ROOT, "tests", "golden", "lut_T07_16_N6.npz"))
    for bc in (eagb.EA_PBC, eagb.EA_OBC):
        job = eagb.SpJob(L, Lz, d["betas"][:nb], d["cum"][:nb], nrep=4, nwords=1, bc=bc, seeds=SEEDS)
        rng = np.random.default_rng(L)
        diff = planes(L, Lz, rng, (64, 2, nb))
        # words whose sample s differs on the first diff[s] sites of each plane, in an order of its own
        S = rng.integers(0, 1 << 64, (1, Lz, L * L, 4, nb), np.uint64)
        for k in range(2):
            rank = rng.permuted(np.tile(np.arange(L * L), (64, nb, Lz, 1)), axis=-1)
            on = rank < diff[:, k][..., None]                       # [sample][slot][z][site]
            x = (on.astype(np.uint64) << np.arange(64, dtype=np.uint64)[:, None, None, None]).sum(0, dtype=np.uint64)
            S[0, :, :, 2 * k + 1] = S[0, :, :, 2 * k] ^ x.transpose(1, 2, 0)
        job.set_spins(S.reshape(1, Lz * L * L, 4, nb))
        assert np.array_equal(job.plane_overlaps(4)[0], diff)
        C = job.plane_correlations(4, dmax)
        assert np.array_equal(C[..., 2, 2], sign_products(diff, L * L, bc == eagb.EA_PBC, dmax))
        # a vanishing overlap adds nothing to the products with its powers either
        want = analysis.plane_correlations(diff, L * L, bc == eagb.EA_PBC, dmax)
        assert np.allclose(C, want, rtol=0, atol=1e-12)
        job.close()

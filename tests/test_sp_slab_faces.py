"""The slab labelling joins slabs over the bonds whose larger end lies in a
slab's first plane or in the lattice's last: these are all bonds between two
slabs, for every boundary condition, odd and even sizes, and any slab height."""
import numpy as np
import pytest

from test_sp import eagb


@pytest.mark.parametrize("L,Lz", [(2, 3), (3, 4), (3, 7), (4, 9), (5, 5), (5, 12), (6, 8), (7, 13)])
@pytest.mark.parametrize("bc", [eagb.EA_PBC, eagb.EA_OBC])
def test_faces_hold_every_bond_between_slabs(L, Lz, bc):
    nb = eagb.sp_graph(L, Lz, bc)[0]
    site = np.repeat(np.arange(len(nb)), 6)
    hi = np.maximum(site, nb.reshape(-1))
    z = hi // (L * L)
    for D in range(1, Lz + 1):
        across = site // (L * L) // D != nb.reshape(-1) // (L * L) // D
        assert ((z % D == 0) | (z == Lz - 1))[across].all()

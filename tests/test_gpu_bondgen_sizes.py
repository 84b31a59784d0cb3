"""dem_generate_bonds at the edges of its blocks of 64 contact records and of
the host's chunks of 4,096 bonds: bit for bit with the oracle's regen_bonds."""
import numpy as np
import pytest

import dem
import dem_scenes
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,max_bonds", [(1, 6), (63, 14), (64, 1), (65, 6), (4100, 1), (4700, 2)])
def test_sizes_bit_exact(n, max_bonds):
    sc, _, _ = dem_scenes.dense_bed(n, seed=n, spacing=1.9)
    bonds, contacts = dem.generate_bonds(sc["pos"], sc["radii"], max_bonds=max_bonds)
    rb, rc = oracle.regen_bonds(sc["pos"], sc["radii"], max_bonds)
    assert np.array_equal(bonds, rb) and np.array_equal(contacts, rc)
    assert bonds.size // 3 > 4096 or max_bonds != 2, "one chunk only"

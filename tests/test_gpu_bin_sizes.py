"""dem_broad_phase_noalloc at the edges of its blocks, digits and packed words:
whole numbers, equal to numpy's stable sort."""
import numpy as np
import pytest

import dem
from test_zz_no_alloc import _call, _lib, _numpy_broad_phase

pytestmark = pytest.mark.gpu


# no particle, one, a block's first and last elements, chunks and one more;
# 2^23 is the last size whose index shares a word with the second digit.
# Cells: one, the last grid of one digit and the first of two, the largest.
@pytest.mark.parametrize("n", [0, 1, 31, 1023, 1024, 4097, 311297, 1 << 23, (1 << 23) + 1])
@pytest.mark.parametrize("grid", [(1, 1), (73, 7), (16, 32), (511, 513), (262143, 1)])
def test_sizes(n, grid):
    torch = pytest.importorskip("torch")
    if n > 400000 and grid != (511, 513):
        pytest.skip("one grid for the largest sizes")
    gw, gh = grid
    rng = np.random.default_rng(n % 1000 + gw)
    pr = np.zeros((n, 4), np.float32)
    pr[:, 0] = rng.uniform(-0.05, 1.05, n) * gw
    pr[:, 1] = rng.uniform(-0.05, 1.05, n) * gh
    pr[:, 2] = rng.random(n) > 0.01
    if n > 5000:  # one crowded cell
        pr[n // 3: n // 2, :2] = (0.5, 0.5)
    g = (0.0, 0.0, 1.0, gw, gh)
    keys, order, cs = _call(_lib(), torch, torch.device("cuda", 0), pr, g)
    nk, no, ncs = _numpy_broad_phase(pr, *g)
    assert np.array_equal(keys, nk) and np.array_equal(order, no) and np.array_equal(cs, ncs)

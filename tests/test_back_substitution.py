"""The RREF's back substitution over pairs of diagonal blocks: ranks around the number of blocks from which
pairs are formed (eight blocks of 128, then of 256), odd numbers of blocks, last blocks of one row and of a whole block."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [2, 13, 65521, 2147483629, 4294967291])
@pytest.mark.parametrize("r", [896, 897, 1025, 1153, 2050])
def test_pairs_of_blocks(engine, p, r):
    rng = np.random.default_rng(r)
    n = r + 41
    A = rng.integers(0, p, (r, n), dtype=np.uint64).astype(np.uint32)
    A[:, 5] = 0  # a free column among the pivots
    R, piv = O.rref(p, A)[:2]
    got, gpiv = engine.rref(p, A)[:2]
    assert list(gpiv) == list(piv)
    assert np.array_equal(got, R)

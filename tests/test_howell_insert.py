"""The Howell pass by insertion of the non-zero closures, and the blocked reduce-above, against the oracle:
forms with many closures, displaced pivots, columns without a pivot, and sizes around the reduce block."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _same(engine, ell, k, A):
    H1, c1, v1 = engine.howell(ell, k, A)
    H2, c2, v2 = O.howell(ell, k, A)
    assert np.array_equal(c1, c2) and np.array_equal(v1, v2) and np.array_equal(H1, H2)


@pytest.mark.parametrize("ell,k", [(2, 2), (2, 16), (2, 31), (3, 4), (3, 20), (7, 3)])
@pytest.mark.parametrize("m,n", [(1, 1), (3, 40), (40, 3), (63, 64), (64, 66), (65, 130), (150, 150)])
def test_many_closures(engine, ell, k, m, n):
    q = ell ** k
    rng = np.random.default_rng(m * 100 + n + k)
    A = rng.integers(0, q, (m, n), dtype=np.uint64)
    # every row divisible by a power of ell: dense rows with non-unit pivots, so dense non-zero closures
    e = rng.integers(0, k, m)
    _same(engine, ell, k, (A * (np.uint64(ell) ** e.astype(np.uint64))[:, None] % np.uint64(q)).astype(np.uint32))
    # and column gaps: pivots missing, closures landing on empty columns
    A[:, rng.permutation(n)[: n // 3]] = 0
    e = np.minimum(rng.geometric(0.4, m) - 1, k - 1)
    B = (A * (np.uint64(ell) ** e.astype(np.uint64))[:, None] % np.uint64(q)).astype(np.uint32)
    _same(engine, ell, k, B)
    _same(engine, ell, k, np.triu(B) if m > 1 else B)


def test_known_answer(engine):
    H, c, v = engine.howell(2, 2, np.array([[2, 1]], np.uint32))  # over Z/4 the closure 2 (2, 1) = (0, 2) is a row
    assert H.tolist() == [[2, 1], [0, 2]] and c.tolist() == [0, 1] and v.tolist() == [1, 1]


def test_thousands_of_pending_rows(engine):
    """More closures on one column than the insertion lists at once."""
    ell, k, n = 2, 3, 1500
    A = np.zeros((n, n), np.uint32)
    A[np.arange(n - 2), np.arange(n - 2)] = 2
    A[: n - 2, n - 2] = 1 + np.arange(n - 2) % 7
    A[: n - 2, n - 1] = np.arange(n - 2) % 8
    _same(engine, ell, k, A)


@pytest.mark.parametrize("ell,k", [(2, 16), (2, 31), (3, 10)])
def test_pivots_that_change(engine, ell, k):
    """Triangular with random valuations on the diagonal: most echelon pivots are displaced by the closures of
    the columns before them, and their own closures with them."""
    n, q = 160, ell ** k
    rng = np.random.default_rng(k)
    A = np.triu(rng.integers(0, q, (n, n), dtype=np.uint64))
    A[np.arange(n), np.arange(n)] = np.array([ell ** int(e) for e in rng.integers(0, k, n)], np.uint64)
    _same(engine, ell, k, A.astype(np.uint32))
    A[:, 10::7] = A[:, 10::7] * ell % q  # no unit in these columns
    _same(engine, ell, k, A.astype(np.uint32))

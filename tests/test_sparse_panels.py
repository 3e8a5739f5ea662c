"""Panels with few non-zero rows (the compact kernel) and the Smith levels' one elimination with left-out
columns, against the oracle: densities that take the compact kernel, its edge of 256 rows, the searching
kernel, and changes between them within one matrix."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _sparse(rng, m, n, per_row, q):
    A = np.zeros((m, n), np.uint32)
    for i in range(m):
        c = rng.integers(0, n, per_row)
        A[i, c] = rng.integers(0, q, per_row, dtype=np.uint64)
    return A


def _mixes(rng, m, n, q):
    yield _sparse(rng, m, n, 2, q)
    B = np.zeros((m, n), np.uint32)                      # near the diagonal, with empty rows and columns
    r = np.arange(min(m, n))
    B[r, r] = rng.integers(0, q, len(r), dtype=np.uint64)
    B[r[:-1], r[1:]] = rng.integers(0, min(3, q), len(r) - 1) if len(r) > 1 else 0
    B[rng.permutation(m)[: m // 4]] = 0
    yield B
    C = _sparse(rng, m, n, 1, q)                         # a dense stripe: from few rows to all of them and back
    C[:, n // 3: n // 3 + min(40, n // 3)] = rng.integers(0, q, (m, min(40, n // 3)), dtype=np.uint64)
    yield C


@pytest.mark.parametrize("p", [2, 3, 251, 65521, 2147483629, 4294967291])
@pytest.mark.parametrize("m,n", [(1, 1), (40, 300), (256, 256), (257, 300), (600, 500)])
def test_fields(engine, p, m, n):
    rng = np.random.default_rng(m + n + p % 101)
    for A in _mixes(rng, m, n, p):
        R1, p1 = engine.rref(p, A)
        R2, p2 = O.rref(p, A)
        assert np.array_equal(p1, p2) and np.array_equal(R1, R2)
        k = min(m, n)
        D = A[:k, :k].copy()
        D[np.arange(k), rng.permutation(k)] = 1
        assert engine.det(p, D) == O.det(p, D)


@pytest.mark.parametrize("rows", [255, 256, 257])
def test_the_list_is_full(engine, rows):
    """Panels whose non-zero rows just fit the compact kernel, or just do not."""
    rng = np.random.default_rng(rows)
    A = np.zeros((700, 200), np.uint32)
    A[rng.permutation(700)[:rows]] = rng.integers(0, 13, (rows, 200))
    for p in (13, 65521):
        R1, p1 = engine.rref(p, A)
        R2, p2 = O.rref(p, A)
        assert np.array_equal(p1, p2) and np.array_equal(R1, R2)


@pytest.mark.parametrize("ell,k", [(2, 1), (2, 16), (2, 31), (3, 10), (3, 20), (5, 3), (65521, 1)])
@pytest.mark.parametrize("m,n", [(1, 1), (70, 64), (64, 130), (300, 300), (700, 400)])
def test_rings(engine, ell, k, m, n):
    q = ell ** k
    rng = np.random.default_rng(m + n + k)
    for A in _mixes(rng, m, n, q):
        e = np.minimum(rng.geometric(0.5, m) - 1, k - 1).astype(np.uint64)
        A = (A.astype(np.uint64) * (np.uint64(ell) ** e)[:, None] % np.uint64(q)).astype(np.uint32)
        assert np.array_equal(engine.smith(ell, k, A), O.smith(ell, k, A))
        H1, c1, v1 = engine.howell(ell, k, A)
        H2, c2, v2 = O.howell(ell, k, A)
        assert np.array_equal(c1, c2) and np.array_equal(v1, v2) and np.array_equal(H1, H2)


@pytest.mark.parametrize("ell,k", [(2, 8), (3, 5)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_dense_levels(engine, ell, k, mode):
    """Dense level matrices with many columns left out (search over a cluster), and the two-elimination
    form of a level (the grid kernel)."""
    q = ell ** k
    rng = np.random.default_rng(k)
    A = rng.integers(0, q, (400, 330), dtype=np.uint64)
    A[:, rng.permutation(330)[:150]] *= np.uint64(ell)
    A[:, rng.permutation(330)[:60]] *= np.uint64(ell)
    A = (A % np.uint64(q)).astype(np.uint32)
    B = O.gemm(q, A[:, :200], rng.integers(0, q, (200, 330), dtype=np.uint64).astype(np.uint32))
    try:
        engine.set_panel_kernel(mode)
        for M in (A, B, (B.astype(np.uint64) * ell % q).astype(np.uint32)):
            assert np.array_equal(engine.smith(ell, k, M), O.smith(ell, k, M))
    finally:
        engine.set_panel_kernel(0)


@pytest.mark.parametrize("rows", [31, 32, 33, 64, 65, 127, 128, 129])
def test_the_edges_of_the_list(engine, rows):
    """Panels whose non-zero rows fill the compact kernel's warps, or its list, or one row more."""
    rng = np.random.default_rng(rows)
    for p in (2, 13, 65521, 2147483629):
        A = np.zeros((400, 200), np.uint32)
        A[np.sort(rng.permutation(400)[:rows])] = rng.integers(0, p, (rows, 200))
        A[:, 70:120] = 0
        A[rng.permutation(400)[: rows // 2], 80] = 1
        R1, p1 = engine.rref(p, A)
        R2, p2 = O.rref(p, A)
        assert np.array_equal(p1, p2) and np.array_equal(R1, R2)


@pytest.mark.parametrize("ell,k", [(2, 4), (2, 31), (3, 10)])
@pytest.mark.parametrize("m,n", [(130, 300), (300, 200), (200, 400)])
def test_levels_that_end_early(engine, ell, k, m, n):
    """Level matrices whose units are all in the first columns, the rest of them multiples of ell or zero (the
    elimination ends when no unit is left, and the rest is the next level's), or in a few late ones."""
    q = ell ** k
    rng = np.random.default_rng(m + n + k)
    A = rng.integers(0, q, (m, n), dtype=np.uint64)
    rows = (np.uint64(ell) ** rng.integers(0, k, m).astype(np.uint64))[:, None]
    late = A.copy()
    late[:, : n - 20] *= np.uint64(ell)
    zero = A * rows % np.uint64(q)
    zero[:, 100:] = 0
    first = A * np.uint64(ell)
    first[:, :30] = A[:, :30]
    for M in (A * rows, zero, late, first, late * rows):
        M = (M % np.uint64(q)).astype(np.uint32)
        assert np.array_equal(engine.smith(ell, k, M), O.smith(ell, k, M))


@pytest.mark.parametrize("ell,k", [(2, 8), (3, 5)])
def test_level_flags_of_many_rows(engine, ell, k):
    """More rows than the look over a level has CTAs: zero, then multiples of ell, then one unit at the end; and
    each of them everywhere."""
    m, n, q = 3000, 40, ell ** k
    rng = np.random.default_rng(k)
    unit = np.zeros((m, n), np.uint32)
    unit[m // 3:] = rng.integers(0, q // ell, (m - m // 3, n)) * ell
    unit[m - 1, n - 1] = 1
    dense = rng.integers(0, q, (m, n), dtype=np.uint64).astype(np.uint32)
    for M in (unit, np.where(unit == 1, 0, unit), dense, np.zeros((m, n), np.uint32)):
        assert np.array_equal(engine.smith(ell, k, M), O.smith(ell, k, M))

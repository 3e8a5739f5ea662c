"""The top-block path: the in-place fraction-free Gauss-Jordan inversion with its row moves as exact integer
arithmetic (CPU), and the device eliminations at the sizes where the path's row slots, spare rows and
early end lie (GPU, against the oracle)."""
import random

import numpy as np
import pytest

import oracle as O


def _block_inverse(A, q, rho, unit, nb, sub):
    """panel_block_kernel in Python integers, sub-panels of `sub` columns: (pivot rows, inverse of the pivot
    block in pivot order, pivots), or None."""
    T = [list(r) for r in A]
    rows, w = len(T), len(T[0])
    pivoted, order, diag, V = set(), [], [], 1
    for cs in range(0, nb, sub):
        cols = range(cs, min(cs + sub, nb))
        S, scale, mine = 1, [], []
        for t in cols:
            prow = next((i for i in range(rows) if i not in pivoted and unit(T[i][t])), None)
            if prow is None:
                return None
            pivoted.add(prow)
            mine.append(prow)
            scale.append(S)
            x, pr = [T[i][t] for i in range(rows)], list(T[prow])
            diag.append(x[prow] * pow(S * V, -1, q) % q)
            for i in range(rows):
                for j in cols:
                    y, p = (0, S) if j == t else (T[i][j], pr[j])
                    T[i][j] = (S if j == t else T[i][j]) if i == prow else (x[prow] * y - x[i] * p) * rho % q
            S = S * x[prow] * rho % q
        P = [list(T[i]) for i in mine]
        for k, i in enumerate(mine):
            for j in cols:
                T[i][j] = T[i][j] * scale[k] * V * rho % q
        for i in range(rows):
            C = [T[i][j] for j in cols]
            for j in range(w):
                if j in cols:
                    T[i][j] = T[i][j] * V * rho * rho % q
                else:
                    y = 0 if i in mine else S * T[i][j]
                    T[i][j] = (y + sum(c * p[j] for c, p in zip(C, P))) * rho * rho % q
        V = V * S * rho * rho % q
        order += mine
    vinv = pow(V, -1, q)
    return order, [[T[i][s] * vinv % q for s in range(w)] for i in order], diag


@pytest.mark.parametrize("q,ell", [(2, 2), (3, 3), (13, 13), (65521, 65521), (1 << 16, 2), (3 ** 10, 3)])
def test_gauss_jordan_model(q, ell):
    rnd = random.Random(q)
    rho = pow(pow(2, 32), -1, q) if q % 2 else 1
    done = 0
    for _ in range(80):
        nb, extra = rnd.randint(1, 9), rnd.choice([0, 0, 1, 3])  # extra: columns beyond the pivots (no spare rows)
        A = [[rnd.randrange(q) for _ in range(nb + extra)] for _ in range(nb if extra else nb + rnd.randint(0, 6))]
        got = _block_inverse(A, q, rho, lambda x: x % ell != 0, nb, 4)
        if got is None:
            continue
        order, M, diag = got
        B = [A[i][:nb] for i in order]
        for j in range(nb + extra):  # M[:, :nb] B = I, M[:, :nb] A[order, nb:] = M[:, nb:]
            col = [sum(M[i][c] * A[order[c]][j] for c in range(nb)) % q for i in range(nb)]
            assert col == ([int(i == j) for i in range(nb)] if j < nb else [M[i][j] for i in range(nb)])
        det, Z = 1, [list(r) for r in B]
        for t in range(nb):  # the pivots are those of the elimination without scales
            det = diag[t]
            assert Z[t][t] % q == det
            inv = pow(det, -1, q)
            for i in range(t + 1, nb):
                f = Z[i][t] * inv % q
                Z[i] = [(y - f * p) % q for y, p in zip(Z[i], Z[t])]
        done += 1
    assert done > 15


def _rand(rng, shape, p):
    return rng.integers(0, p, shape, dtype=np.uint64).astype(np.uint32)


# rows around the row slots (64, 96, 128) and the panel widths, p on both sides of the dispatch's lines
@pytest.mark.gpu
@pytest.mark.parametrize("p", [2, 3, 13, 251, 257, 8179, 8191, 8209, 1048573, 1048583, 2147483629, 4294967291])
@pytest.mark.parametrize("m,n", [(1, 5), (63, 64), (64, 65), (65, 64), (95, 200), (96, 96), (97, 130), (129, 70), (200, 333)])
def test_block_slots(engine, p, m, n):
    rng = np.random.default_rng(m * 1000 + n + p % 97)
    A = _rand(rng, (m, n), p)
    r = max(1, min(m, n) * 2 // 3)
    D = O.gemm(p, _rand(rng, (m, r), p), _rand(rng, (r, n), p))  # rank-deficient: the early end
    P = np.zeros((m, n), np.uint32)                              # scattered units only: every pivot row moves
    P[rng.permutation(m)[: min(m, n)], rng.permutation(n)[: min(m, n)]] = 1
    Z = np.zeros((m, n), np.uint32)
    for M in (A, D, P, Z):
        R1, p1 = engine.rref(p, M)
        R2, p2 = O.rref(p, M)
        assert np.array_equal(p1, p2) and np.array_equal(R1, R2)


@pytest.mark.gpu
@pytest.mark.parametrize("p", [3, 13, 65521, 2147483629])
@pytest.mark.parametrize("n", [2, 33, 64, 100, 257])
def test_determinant_sign_of_row_moves(engine, p, n):
    rng = np.random.default_rng(n)
    for _ in range(3):
        perm = rng.permutation(n)
        M = np.zeros((n, n), np.uint32)
        M[np.arange(n), perm] = 1
        assert engine.det(p, M) == O.det(p, M)
        A = _rand(rng, (n, n), p)[perm]
        assert engine.det(p, A) == O.det(p, A)


@pytest.mark.gpu
@pytest.mark.parametrize("ell,k", [(2, 1), (2, 16), (2, 31), (3, 5), (3, 20), (5, 3)])
@pytest.mark.parametrize("m,n", [(64, 64), (97, 130), (200, 100)])
def test_rings_dense(engine, ell, k, m, n):
    """Dense matrices over Z/ell^k: unit pivots abound, so the top block settles the panels."""
    q = ell ** k
    rng = np.random.default_rng(m + k)
    A = _rand(rng, (m, n), q)
    H1, c1, v1 = engine.howell(ell, k, A)
    H2, c2, v2 = O.howell(ell, k, A)
    assert np.array_equal(H1, H2) and np.array_equal(c1, c2) and np.array_equal(v1, v2)
    assert np.array_equal(engine.smith(ell, k, A), O.smith(ell, k, A))


@pytest.mark.gpu
@pytest.mark.parametrize("p", [65521, 2147483629, 4294967291])
@pytest.mark.parametrize("panel", [0, 1, 2, 3, 5])
def test_queued_panels_stand_still(engine, p, panel):
    """A panel that the host had expected the top block to settle, met while the work behind it is queued:
    a column without a pivot, a pivot row out of order, and both in neighbouring panels."""
    rng = np.random.default_rng(panel)
    n = 450
    for kind in range(3):
        A = _rand(rng, (n, n), p)
        c = 64 * panel + 17
        if kind != 1:
            A[:, c] = O.gemm(p, A[:, :c], _rand(rng, (c, 1), p))[:, 0]  # dependent on the columns before it
        if kind != 0 and panel > 0:
            A[c + 40] = A[c - 60]                                      # a zero on the diagonal further down
        R1, p1 = engine.rref(p, A)
        R2, p2 = O.rref(p, A)
        assert np.array_equal(p1, p2) and np.array_equal(R1, R2)
        assert engine.det(p, A) == O.det(p, A)

"""The device memory that an elimination takes beside its matrix."""
import numpy as np
import pytest

import hacs_b200
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [65521, 2147483629])
def test_tall_matrix_takes_little_beside_it(p):
    """2^20 x 48, few non-zero rows and then all: two left factors W of the matrix's size (48 columns, not a whole
    panel's 64) with an eighth of headroom, and scratch that does not grow with the rows."""
    import torch

    m, n = 1 << 20, 48
    torch.cuda.empty_cache()
    A = torch.zeros((m, n), dtype=torch.int32, device="cuda")
    A[:: m // 64] = torch.randint(0, p, (64, n), dtype=torch.int32, device="cuda")
    A[:, 40:].random_(0, p)
    W = A.clone()
    with hacs_b200.Engine(0) as warm:  # the kernels are loaded
        warm.use_torch_stream()
        warm.rref_dev(p, W[:1000].clone())
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    with hacs_b200.Engine(0) as eng:
        eng.use_torch_stream()
        free = torch.cuda.mem_get_info()[0]
        piv = eng.rref_dev(p, W)
        taken = free - torch.cuda.mem_get_info()[0]
        assert taken < 2.75 * 4 * m * n, taken / (4 * m * n)
    assert list(piv) == list(range(n))
    assert torch.equal(W[:n], torch.eye(n, dtype=torch.int32, device="cuda")) and not bool(W[n:].any())


@pytest.mark.parametrize("cols", [5, 31, 63, 64, 65, 100, 129])
def test_few_columns(engine, cols):
    """Panels narrower than 64 columns and the first panels behind them, near-empty and dense ones in turn."""
    rng = np.random.default_rng(cols)
    for p in (13, 65521, 2147483629):
        for rows in (40, 300):
            A = np.where(rng.random((rows, cols)) < 0.03, rng.integers(1, p, (rows, cols)), 0).astype(np.uint32)
            for M in (A, np.hstack([A, rng.integers(0, p, (rows, 7), dtype=np.uint64).astype(np.uint32), A])):
                R1, p1 = engine.rref(p, M)
                R2, p2 = O.rref(p, M)
                assert np.array_equal(p1, p2) and np.array_equal(R1, R2)

"""Long-row matrix-vector products: lengths around the columns that a CTA keeps
of x (2048, 4096, 8192, and several passes), few and many rows, aligned and
unaligned rows, strided vectors, the three ops."""
import numpy as np
import pytest

import hacs_b200
from oracle import level12 as L12

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [2, 65521, 2147483629, 4294967291])
@pytest.mark.parametrize("k", [2048, 2049, 4096, 4100, 8191, 8192, 8196, 16381, 20001])
def test_long_rows(engine, p, k):
    import torch

    rng = np.random.default_rng(k)
    for m, pad, xs, op in [(1, 0, 1, hacs_b200.SET), (3, 4, 1, hacs_b200.ADD), (7, 1, 1, hacs_b200.SUB),
                           (5, 0, 3, hacs_b200.ADD), (1300, 0, 1, hacs_b200.SUB), (2501, 0, 1, hacs_b200.ADD)]:
        A = rng.integers(0, p, (m, k + pad), dtype=np.uint64).astype(np.uint32)
        x = rng.integers(0, p, (k * xs,), dtype=np.uint64).astype(np.uint32)
        y = rng.integers(0, p, (m,), dtype=np.uint64).astype(np.uint32)
        A[0] = p - 1
        dA, dx, dy = (torch.from_numpy(v.view(np.int32)).cuda() for v in (A, x, y))
        torch.cuda.synchronize()
        engine.gemv_dev(p, dA[:, :k], dx[::xs], dy, op)
        engine.sync()
        want = L12.gemv(p, A[:, :k], x[::xs], y, op)
        assert np.array_equal(dy.cpu().numpy().view(np.uint32), want), (m, pad, xs, op)

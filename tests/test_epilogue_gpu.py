"""The limb GEMM's epilogue and its one-k-block pipeline at their edges, against the oracle (exact)."""
import numpy as np
import pytest

import oracle as O
from hacs_b200 import ADD, SET, SUB

pytestmark = pytest.mark.gpu


# moduli on both sides of each limb count and of the 32-bit reduction's range; K around the one-k-block
# widths and the exact-accumulation chunk (all entries p - 1 give the largest sums)
@pytest.mark.parametrize("p", [2, 128, 255, 256, 257, 511, 65535, 65537, 131071, 131073, (1 << 24) - 1, (1 << 24) + 43,
                               (1 << 25) + 1, (1 << 31) - 1, (1 << 31) + 11, (1 << 32) - 5])
@pytest.mark.parametrize("k", [1, 32, 33, 64, 65, 128, 129, 8192])
def test_epilogue_extreme_sums(engine, p, k):
    m, n = 130, 83
    A = np.full((m, k), p - 1, np.uint32)
    B = np.full((k, n), p - 1, np.uint32)
    A[::3] = 1
    B[:, ::5] = p // 2
    C = (np.arange(m * n, dtype=np.uint64) * 2654435761 % p).astype(np.uint32).reshape(m, n)
    for op in (SET, ADD, SUB):
        assert np.array_equal(engine.gemm(p, A, B, C, op), O.gemm(p, A, B, C, op)), op


# C windows with and without 16-byte rows, widths with every remainder of a 16-byte piece, several tile
# columns per CTA and several CTAs per column
@pytest.mark.parametrize("p", [13, 65521, 16777213, 2147483629])
@pytest.mark.parametrize("m,n,k,ld,off", [(300, 257, 64, 260, 0), (300, 258, 64, 261, 0), (129, 259, 32, 264, 1),
                                          (2500, 515, 64, 516, 0), (1, 3, 100, 4, 0), (140, 4100, 17, 4101, 2)])
def test_one_k_block_windows(engine, p, m, n, k, ld, off):
    import torch

    rng = np.random.default_rng(m + n + k)
    A, B = (rng.integers(0, p, s, dtype=np.uint64).astype(np.uint32) for s in ((m, k), (k, n)))
    C = rng.integers(0, p, (m, n), dtype=np.uint64).astype(np.uint32)
    dA, dB = (torch.from_numpy(x.view(np.int32)).cuda() for x in (A, B))
    buf = torch.full((m * ld + off,), 7, dtype=torch.int32, device="cuda")
    win = buf[off:].view(m, ld)[:, :n]
    engine.use_torch_stream()
    for op in (ADD, SUB):
        win.copy_(torch.from_numpy(C.view(np.int32)).cuda())
        engine.gemm_dev(p, dA, dB, win, op)
        torch.cuda.synchronize()
        assert np.array_equal(win.cpu().numpy().view(np.uint32), O.gemm(p, A, B, C, op)), op
        assert (buf[off:].view(m, ld)[:, n:] == 7).all()
    engine.use_own_stream()

"""The products over the 8-bit residue system (u64 entries, and u32 entries where they pay) at the edges of
their plans: moduli counts, the largest sums, ragged tiles, several chunks of K; against exact integers."""
import numpy as np
import pytest

import oracle as O
from hacs_b200 import ADD, SET, SUB

pytestmark = pytest.mark.gpu


def _exact(A, B, p):
    """A B mod p in Python integers through a few float-free object dot products."""
    return np.array((A.astype(object) @ B.astype(object)) % p, dtype=object)


@pytest.mark.parametrize("p", [(1 << 32) + 15, (1 << 40) - 87, (1 << 61) - 1, (1 << 63) - 25, (1 << 63) + 29, (1 << 64) - 59, 1 << 40])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (5, 33, 32), (130, 129, 65), (3, 260, 700)])
def test_u64_extremes(engine, p, m, n, k):
    rng = np.random.default_rng(m + n + k)
    A = rng.integers(0, p, (m, k), dtype=np.uint64)
    B = rng.integers(0, p, (k, n), dtype=np.uint64)
    A[::2] = p - 1
    B[:, ::3] = p - 1
    C = rng.integers(0, p, (m, n), dtype=np.uint64)
    want = _exact(A, B, p)
    for op, w in ((SET, want), (ADD, (C.astype(object) + want) % p), (SUB, (C.astype(object) - want) % p)):
        assert (engine.gemm_u64(p, A, B, C, op).astype(object) == w).all(), op


def test_u64_several_chunks_of_k(engine):
    p, k = (1 << 61) - 1, 33024 + 700
    A = np.full((3, k), p - 1, np.uint64)
    B = np.full((k, 40), p - 1, np.uint64)
    B[:, 1] = 12345
    want = [k % p if j != 1 else (p - 12345 * k % p) % p for j in range(40)]
    assert (engine.gemm_u64(p, A, B) == np.array(want, np.uint64)).all()


# shapes that the u32 dispatch sends to the residue system (few tiles, long K), and moduli on both sides of 2^31
@pytest.mark.parametrize("p", [(1 << 24) + 43, 134217757, 2147483629, 4294967291])
@pytest.mark.parametrize("m,n,k", [(64, 64, 8192), (70, 131, 9001), (300, 257, 8000)])
def test_u32_long_k(engine, p, m, n, k):
    import torch

    rng = np.random.default_rng(k)
    A = rng.integers(0, p, (m, k), dtype=np.uint64).astype(np.uint32)
    B = rng.integers(0, p, (k, n), dtype=np.uint64).astype(np.uint32)
    A[::2] = p - 1
    B[:, ::3] = p - 1
    C = rng.integers(0, p, (m, n), dtype=np.uint64).astype(np.uint32)
    dA, dB = (torch.from_numpy(x.view(np.int32)).cuda() for x in (A, B))
    buf = torch.full((m, n + 3), 7, dtype=torch.int32, device="cuda")
    engine.use_torch_stream()
    try:
        for op in (SET, ADD, SUB):
            buf[:, :n].copy_(torch.from_numpy(C.view(np.int32)).cuda())
            engine.gemm_dev(p, dA, dB, buf[:, :n], op)
            torch.cuda.synchronize()
            assert np.array_equal(buf[:, :n].cpu().numpy().view(np.uint32), O.gemm(p, A, B, C, op)), op
            assert (buf[:, n:] == 7).all()
    finally:
        engine.use_own_stream()


def test_captured_product_without_room_for_the_residue_planes():
    """A context warmed with limb products only: a capture cannot grow the planes to what the residue system
    takes, so the captured product takes the limb route; outside the capture it may take the other.  Both agree."""
    import torch

    import hacs_b200
    from hacs_b200 import _lib

    p, n = 2147483629, 3072
    s = torch.cuda.Stream()
    with hacs_b200.Engine(0) as eng, torch.cuda.stream(s):
        eng.use_torch_stream()
        A, B = (torch.randint(0, p, (n, n), dtype=torch.int32, device="cuda") for _ in range(2))
        C = [torch.zeros((n, n), dtype=torch.int32, device="cuda") for _ in range(3)]
        assert _lib.lib().hme_ctx_set_gemm_variant(eng._h, 0) == 0
        eng.gemm_dev(p, A, B, C[0])
        assert _lib.lib().hme_ctx_set_gemm_variant(eng._h, -1) == 0
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            eng.gemm_dev(p, A, B, C[1])
        graph.replay()
        torch.cuda.synchronize()
        eng.gemm_dev(p, A, B, C[2])
        torch.cuda.synchronize()
        assert torch.equal(C[0], C[1]) and torch.equal(C[0], C[2])

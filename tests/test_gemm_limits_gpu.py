"""Products at the limits of their index arithmetic: planes whose stacked rows pass a 32-bit coordinate, empty
operands, dimensions that are refused."""
import numpy as np
import pytest

import hacs_b200
from hacs_b200 import _lib

pytestmark = pytest.mark.gpu

P31 = 2147483629


def _room(gb):
    import torch

    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < gb << 30:
        pytest.skip(f"needs {gb} GB of device memory")


@pytest.mark.parametrize("p,wide", [((1 << 40) - 87, True), (P31, False)])
def test_planes_beyond_a_32_bit_coordinate(p, wide):
    """1 x 1 x n: the residue planes of B stack to t n > 2^31 rows (t = 11 moduli of n = 200 000 000 columns with
    64-bit entries, t = 9 of 240 000 000 with 32-bit ones)."""
    import torch

    _room(100)
    n, a = (200_000_000, 12345) if wide else (240_000_000, 1234567)
    kind = torch.int64 if wide else torch.int32
    A = torch.full((1, 1), a, dtype=kind, device="cuda")
    B = torch.empty((1, n), dtype=kind, device="cuda").random_(0, p, generator=torch.Generator("cuda").manual_seed(n))
    C = torch.full((1, n), 7, dtype=kind, device="cuda")
    with hacs_b200.Engine(0) as eng:
        eng.use_torch_stream()
        (eng.gemm_u64_dev if wide else eng.gemm_dev)(p, A, B, C)
        torch.cuda.synchronize()
        for c0 in range(0, n, 20_000_000):
            s = slice(c0, min(n, c0 + 20_000_000))
            assert torch.equal(C[0, s].to(torch.int64), B[0, s].to(torch.int64) * a % p), c0


@pytest.mark.parametrize("m,n,k", [(0, 4096, 4096), (4096, 0, 4096), (0, 0, 4096)])
def test_empty_product_touches_nothing(m, n, k):
    """No rows (or columns) and non-null pointers: C is left alone, as by every other modulus and size."""
    import torch

    L = _lib.lib()
    A = torch.ones((1, 4096), dtype=torch.int32, device="cuda")
    B = torch.ones((4096, 4096), dtype=torch.int32, device="cuda")
    C = torch.full((8, 4096), 7, dtype=torch.int32, device="cuda")
    with hacs_b200.Engine(0) as eng:
        eng.use_torch_stream()
        for p in (65521, P31):
            for op in (hacs_b200.SET, hacs_b200.ADD, hacs_b200.SUB):
                assert L.hme_gemm_u32_dev(eng._h, p, m, n, k, A.data_ptr(), 4096, B.data_ptr(), 4096, C.data_ptr(),
                                          4096, op) == _lib.HME_OK
            assert L.hme_schur_update_u32_dev(eng._h, p, m, n, k, A.data_ptr(), 4096, B.data_ptr(), 4096,
                                              C.data_ptr(), 4096) == _lib.HME_OK
        torch.cuda.synchronize()
    assert bool((C == 7).all())


def test_refused_products_stay_refused():
    """A side of 2^30 or more, a leading dimension below the row, an unknown op: HME_EINVAL before anything runs.
    (The pointers are never followed.)"""
    import torch

    L = _lib.lib()
    t = torch.ones(64, dtype=torch.int32, device="cuda").data_ptr()
    with hacs_b200.Engine(0) as eng:
        for m, n, k, lda, ldb, ldc, op in ((1, 1, 1 << 30, 1 << 30, 1, 1, 0), (1, 1 << 30, 1, 1, 1 << 30, 1 << 30, 0),
                                           (1 << 30, 1, 1, 1, 1, 1, 0), (64, 64, 8192, 8191, 64, 64, 0),
                                           (64, 64, 8192, 8192, 63, 64, 0), (64, 64, 8192, 8192, 64, 63, 0),
                                           (64, 64, 8192, 8192, 64, 64, 3)):
            assert L.hme_gemm_u32_dev(eng._h, P31, m, n, k, t, lda, t, ldb, t, ldc, op) == _lib.HME_EINVAL
        assert L.hme_gemm_u64_dev(eng._h, (1 << 61) - 1, 1, (1 << 32) - 1, 1, t, 1, t, (1 << 32) - 1, t, (1 << 32) - 1,
                                  0) == _lib.HME_EINVAL


def test_matrix_vector_product_of_the_longest_rows():
    """Rows of 2^30 + 5 columns (the first beyond one piece), rows of 2^32 - 1 columns and 2^32 - 1 rows: the
    latter two as views of stride 0."""
    import torch

    L, most = _lib.lib(), (1 << 32) - 1
    _room(24)
    with hacs_b200.Engine(0) as eng:
        eng.use_torch_stream()

        def gemv(p, m, k, A, a_rs, a_cs, x, x_rs, y, op):
            assert L.hme_gemv_u32_dev(eng._h, p, m, k, A.data_ptr(), a_rs, a_cs, x.data_ptr(), x_rs, y.data_ptr(), 1,
                                      op) == _lib.HME_OK
            torch.cuda.synchronize()

        k, p = (1 << 30) + 5, 65521
        x, A = (torch.empty(k, dtype=torch.int32, device="cuda").random_(0, p) for _ in range(2))
        dot = sum(int((A[c:c + (1 << 28)].to(torch.int64) * x[c:c + (1 << 28)]).sum()) for c in range(0, k, 1 << 28))
        for op, want in ((hacs_b200.SET, dot), (hacs_b200.ADD, 11 + dot), (hacs_b200.SUB, 11 - dot)):
            y = torch.full((1,), 11, dtype=torch.int32, device="cuda")
            gemv(p, 1, k, A, k, 1, x, 1, y, op)
            assert int(y[0]) == want % p
        del x, A
        torch.cuda.empty_cache()
        a, b = (torch.full((1,), v, dtype=torch.int32, device="cuda") for v in (P31 - 1, 123456789))
        y = torch.full((3,), 11, dtype=torch.int32, device="cuda")
        gemv(P31, 3, most, a, 0, 0, b, 0, y, hacs_b200.SUB)
        assert y.tolist() == [(11 - (P31 - 1) * 123456789 * most) % P31] * 3
        y = torch.full((most,), 11, dtype=torch.int32, device="cuda")
        gemv(P31, most, 1, a, 0, 1, b, 1, y, hacs_b200.SET)
        assert bool((y == (P31 - 1) * 123456789 % P31).all())

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

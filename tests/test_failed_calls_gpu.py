"""What a call leaves behind when device memory runs out: the context goes on as if the call had not been made.
The allocations that fail here are larger than the device, so they fail whatever else it holds."""
import numpy as np
import pytest

import hacs_b200
import oracle as O
from hacs_b200 import _lib

pytestmark = pytest.mark.gpu

P31 = 2147483629


@pytest.fixture
def eng():
    import torch

    torch.cuda.empty_cache()
    with hacs_b200.Engine(0) as e:
        e.use_torch_stream()
        yield e
    torch.cuda.empty_cache()


def _product_is_right(eng, p=P31, n=200):
    import torch

    rng = np.random.default_rng(n)
    A, B = (rng.integers(0, p, (n, n), dtype=np.uint64).astype(np.uint32) for _ in range(2))
    dA, dB = (torch.from_numpy(x.view(np.int32)).cuda() for x in (A, B))
    dC = torch.full((n, n), 7, dtype=torch.int32, device="cuda")
    eng.gemm_dev(p, dA, dB, dC)
    torch.cuda.synchronize()
    return np.array_equal(dC.cpu().numpy().view(np.uint32), O.gemm(p, A, B))


def test_call_after_a_failed_allocation(eng):
    """A limb product 1 x 1 x 400 000 000 takes 205 GB of planes; the call after it is not refused."""
    import torch

    n = 400_000_000
    A = torch.ones((1, 1), dtype=torch.int32, device="cuda")
    B = torch.ones((1, n), dtype=torch.int32, device="cuda")
    C = torch.empty((1, n), dtype=torch.int32, device="cuda")
    assert _lib.lib().hme_ctx_set_gemm_variant(eng._h, 0) == 0
    with pytest.raises(_lib.HmeError) as e:
        eng.gemm_dev(P31, A, B, C)
    assert e.value.code == _lib.HME_ENOMEM
    assert _product_is_right(eng)

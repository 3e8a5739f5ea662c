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


def test_product_after_an_elimination_that_ran_out_of_memory(eng):
    """The update right of a panel of 65 x 160 000 000 takes 164 GB of planes, with the panel's update queued
    before its outcome is known; the zero in the corner makes the panel raise the flag that queued work obeys."""
    import torch

    if torch.cuda.mem_get_info()[0] < 50 << 30:
        pytest.skip("needs 45 GB of device memory")
    A = torch.zeros((65, 160_000_000), dtype=torch.int32, device="cuda")
    A[:, :64].random_(1, P31)
    A[0, 0] = 0
    with pytest.raises(_lib.HmeError) as e:
        eng.rref_dev(P31, A)
    assert e.value.code == _lib.HME_ENOMEM
    del A
    assert _product_is_right(eng)
    B = np.random.default_rng(3).integers(0, P31, (150, 170), dtype=np.uint64).astype(np.uint32)
    R, piv = eng.rref(P31, B)
    wR, wpiv = O.rref(P31, B)
    assert np.array_equal(R, wR) and list(piv) == list(wpiv)


def test_matrix_is_free_once_its_elimination_has_failed(eng):
    """The panel after the first was launched ahead on a second stream when the update failed: once the call has
    returned its error, nothing writes the matrix any more."""
    import torch

    if torch.cuda.mem_get_info()[0] < 50 << 30:
        pytest.skip("needs 45 GB of device memory")
    A = torch.zeros((65, 160_000_000), dtype=torch.int32, device="cuda")
    for _ in range(3):
        A[:, :256].random_(1, P31)
        with pytest.raises(_lib.HmeError) as e:
            eng.rref_dev(P31, A)
        assert e.value.code == _lib.HME_ENOMEM
        A[:, :256] = 7
        torch.cuda.synchronize()
        assert bool((A[:, :256] == 7).all())

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


def _fill(free):
    """Device memory taken up to `free` bytes."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - free, dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("held", [False, True])
def test_product_beside_full_memory_takes_the_smaller_planes(eng, held):
    """8192^3 mod 2^31 - 19, u = 64 MiB a byte plane, an eighth of headroom on every buffer: the residue system's
    planes take 11.25 u + 22.5 u, the limbs' 4.5 u + 18 u.  With 26 u free, or with the limbs' planes held and
    20 u free, the first does not fit in whole, and the second has to find what it needs."""
    import torch

    n, u = 8192, 8192 * 8192
    L = _lib.lib()
    A, B = (torch.randint(0, P31, (n, n), dtype=torch.int32, device="cuda") for _ in range(2))
    C, want = torch.zeros_like(A), torch.zeros_like(A)
    with hacs_b200.Engine(0) as ref:
        ref.use_torch_stream()
        ref.gemm_dev(P31, A, B, want)
        torch.cuda.synchronize()
    if held:
        assert L.hme_ctx_set_gemm_variant(eng._h, 0) == 0
        eng.gemm_dev(P31, A, B, C)
        assert L.hme_ctx_set_gemm_variant(eng._h, -1) == 0
        C.zero_()
    rest = _fill(20 * u if held else 26 * u)
    try:
        eng.gemm_dev(P31, A, B, C)
        torch.cuda.synchronize()
    finally:
        del rest
    assert torch.equal(C, want)


def test_ranks_beside_full_memory_take_the_smaller_rounds(eng):
    """10000 ranks of 256 x 64 mod 2^31 - 19: rounds of 64 columns take 66.5 + 131 KB a job, rounds of 32 columns
    53 + 65.5 KB (and about 1 KB of tables), an eighth more with headroom.  With 126 KB a job (and the eighth)
    free, between the second and the first one's buffers beside the second one's planes."""
    import torch

    jobs, m, n = 10000, 256, 64
    C = torch.randint(0, P31, (jobs, m, n), dtype=torch.int32, device="cuda")
    C[::3, :, 5] = C[::3, :, 4]
    eng.use_own_stream()
    torch.cuda.synchronize()
    rest = _fill(int(jobs * 126_000 * 1.125))
    try:
        ranks = eng.batch_rank_dev([dict(A=None, B=None, C=C[t], p=P31) for t in range(jobs)])
    finally:
        del rest
    assert (ranks[::3] == n - 1).all() and (ranks[1::3] == n).all() and (ranks[2::3] == n).all()

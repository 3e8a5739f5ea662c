"""The batched rank's rounds of 64 columns (the batch rule): planted, sparse,
shifted and degenerate jobs at the edges of the 64-row block, the 256 listed
rows and the 1024-row limit, odd leading dimensions, one to four limbs; every
rank equals the oracle's and the general schedules'."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _matrices(rng, p):
    def dense(m, n):
        return rng.integers(0, p, (m, n), dtype=np.uint64).astype(np.uint32)

    out = [dense(m, n) for m, n in [(1, 1), (1, 200), (200, 1), (63, 63), (64, 64), (65, 65), (64, 129), (129, 64),
                                    (96, 97), (127, 300), (300, 127), (256, 200), (257, 260), (320, 384)]]
    # planted rank
    for m, n, r in [(64, 64, 63), (128, 128, 64), (200, 260, 65), (300, 300, 1), (400, 300, 256), (1024, 200, 150)]:
        out.append(O.gemm(p, dense(m, r), dense(r, n)))
    # top rows zero, so that the first block has no pivots; leading columns zero; all zero
    A = dense(260, 140)
    A[:100] = 0
    out.append(A)
    A = dense(150, 260)
    A[:, :70] = 0
    out.append(A)
    out.append(np.zeros((80, 90), np.uint32))
    # sparse: banded, a few entries per row, more than 256 rows in a panel
    A = np.zeros((400, 400), np.uint32)
    for i in range(400):
        for j in range(max(0, i - 9), min(400, i + 10)):
            if rng.random() < 0.1:
                A[i, j] = rng.integers(1, p)
    out.append(A)
    out.append(np.where(rng.random((700, 300)) < 0.02, dense(700, 300), 0).astype(np.uint32))
    # every other row a duplicate of the one before
    A = dense(180, 200)
    A[1::2] = A[::2]
    out.append(A)
    # largest residues
    out.append(np.full((70, 130), p - 1, np.uint32))
    A = np.triu(np.full((130, 130), p - 1, np.uint32))
    out.append(A)
    return out


@pytest.mark.parametrize("p", [2, 3, 251, 1021, 65521, 16777213, 2147483647, 4294967291])
def test_rounds_of_64_match_oracle_and_schedules(engine, p):
    import torch

    rng = np.random.default_rng(p % 1000 + 5)
    mats = _matrices(rng, p)
    want = [len(O.rref(p, A)[1]) for A in mats]

    def jobs():
        out = []
        for t, A in enumerate(mats):
            T = torch.zeros((A.shape[0], A.shape[1] + t % 5), dtype=torch.int32, device="cuda")
            T[:, : A.shape[1]] = torch.from_numpy(A.view(np.int32)).cuda()
            out.append({"p": p, "A": None, "B": None, "C": T[:, : A.shape[1]]})
        torch.cuda.synchronize()
        return out

    assert list(engine.batch_rank_dev(jobs())) == want
    # the schedules of 32-column rounds, beside jobs under the batch rule
    rv = np.array([t % 3 - 1 for t in range(len(mats))], dtype=np.int32)
    assert list(engine.batch_rank_dev(jobs(), rank_variants=rv)) == want


def test_rounds_over_several_moduli_and_repeats(engine):
    """Jobs of five moduli and all three panel arithmetics (2, below and above
    2^31) in one call, twice on the same engine."""
    import torch

    rng = np.random.default_rng(11)
    mats = []
    for p in (2, 7, 65521, 2147483629, 4294967291):
        for m, n, r in [(100, 130, 90), (64, 64, 64), (270, 190, 170), (40, 500, 40)]:
            A = rng.integers(0, p, (m, r), dtype=np.uint64).astype(np.uint32)
            B = rng.integers(0, p, (r, n), dtype=np.uint64).astype(np.uint32)
            mats.append((p, O.gemm(p, A, B)))
    want = [len(O.rref(p, A)[1]) for p, A in mats]
    for _ in range(2):
        jobs = [{"p": p, "A": None, "B": None, "C": torch.from_numpy(A.view(np.int32)).cuda()} for p, A in mats]
        torch.cuda.synchronize()
        assert list(engine.batch_rank_dev(jobs)) == want

"""The workloads that the engine's speed is judged by.

Every case is one call (or one short sequence of calls) through
``hacs_b200.Engine``, on inputs a calling program has in hand: device tensors
for the device entry points, numpy arrays for the entry points that take host
matrices.  Sizes and moduli are those of the five benchmark configurations, of
the published timings of the reference engine and of the tests; ``draw`` gives
further cases of the same families.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import hacs_b200
from hacs_b200 import gen
from hacs_b200.stream import DeviceStream

OPS = {"set": hacs_b200.SET, "add": hacs_b200.ADD, "sub": hacs_b200.SUB}
P16, P27, P31, P61 = 65521, 134217757, 2147483629, (1 << 61) - 1

_engines = {}


def _engine(own: bool = False) -> hacs_b200.Engine:
    """The contexts that the program keeps: one on torch's stream, and one on its own
    stream for the job stream, whose rounds are captured in a graph (the legacy
    default stream cannot be captured)."""
    if own not in _engines:
        _engines[own] = hacs_b200.Engine(0)
        if own:
            _engines[own].use_own_stream()
        else:
            _engines[own].use_torch_stream()
    return _engines[own]


def listed():
    return [
        # one small product, odd sides: the call's latency (the side of the reference's batched product)
        {"name": "gemm 129", "op": "gemm", "m": 129, "n": 129, "k": 129, "p": P27, "acc": "set"},
        # configuration 1: the plain modular product
        {"name": "gemm 1024", "op": "gemm", "m": 1024, "n": 1024, "k": 1024, "p": P16, "acc": "set"},
        # a ragged accumulation into C at a 31-bit modulus (the shape of a real boundary block)
        {"name": "gemm ragged add", "op": "gemm", "m": 1677, "n": 771, "k": 1419, "p": P31, "acc": "add"},
        # the large product that the speed-up over the plain method is quoted at
        {"name": "gemm 8192", "op": "gemm", "m": 8192, "n": 8192, "k": 8192, "p": P16, "acc": "set"},
        # 64-bit residues at a Mersenne modulus
        {"name": "gemm_u64 2048", "op": "gemm_u64", "m": 2048, "n": 2048, "k": 2048, "p": P61, "acc": "set"},
        # matrix times vector, as an iteration on one operator does it
        {"name": "gemv 8192", "op": "gemv", "m": 8192, "k": 8192, "p": P31, "acc": "set"},
        # echelon form of a rank-deficient relation matrix (the reference's timed shape)
        {"name": "rref 1677x1419", "op": "rref", "m": 1677, "n": 1419, "rank": 258, "p": P27},
        # configuration 2: echelon form at 31 bits, rank 3900 of 4096
        {"name": "rref 4096", "op": "rref", "m": 4096, "n": 4096, "rank": 3900, "p": P31},
        # a large echelon form over a small field (the reference's timed int8 shape, p = 13)
        {"name": "rref 10515x8668", "op": "rref", "m": 10515, "n": 8668, "rank": 7801, "p": 13},
        # configuration 3: Howell form over Z/2^16
        {"name": "howell 2048", "op": "howell", "n": 2048, "ell": 2, "k": 16},
        # configuration 3: Smith form over Z/3^10
        {"name": "smith 2048", "op": "smith", "n": 2048, "ell": 3, "k": 10},
        # configuration 4: the batched stream, product + rank per job (sides 16 .. 1024)
        {"name": "jobs 2000", "op": "jobs", "count": 2000, "salt": 0x44},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a family with the listed families' weights, sizes uniform in their logarithm."""
    op = rng.choice(["gemm"] * 4 + ["gemm_u64", "gemv"] + ["rref"] * 3 + ["howell", "smith", "jobs"])
    acc = rng.choice(["set", "add", "sub"])
    if op == "gemm":
        m, n, k = (_log_int(rng, 64, 8192) for _ in range(3))
        return {"op": op, "m": m, "n": n, "k": k, "p": rng.choice([251, P16, 16777213, P27, P31, 4294967291]), "acc": acc}
    if op == "gemm_u64":
        m, n, k = (_log_int(rng, 64, 4096) for _ in range(3))
        return {"op": op, "m": m, "n": n, "k": k, "p": rng.choice([(1 << 40) - 87, P61, (1 << 63) - 25]), "acc": acc}
    if op == "gemv":
        return {"op": op, "m": _log_int(rng, 256, 16384), "k": _log_int(rng, 256, 16384),
                "p": rng.choice([251, P16, P27, P31]), "acc": acc}
    if op == "rref":
        m, n = (_log_int(rng, 128, 8192) for _ in range(2))
        r = min(m, n)
        return {"op": op, "m": m, "n": n, "rank": rng.choice([r, rng.randint(1, r), r - r // 20]),
                "p": rng.choice([2, 13, 251, P16, P27, P31])}
    if op in ("howell", "smith"):
        ell, k = rng.choice([(2, 8), (2, 16), (2, 31), (3, 5), (3, 10)])
        return {"op": op, "n": _log_int(rng, 128, 2048), "ell": ell, "k": k}
    return {"op": op, "count": _log_int(rng, 50, 2000), "salt": rng.randrange(1 << 16)}


# ---- inputs --------------------------------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, rows: int, cols: int, p: int) -> torch.Tensor:
    """Uniform residues of Z/p (p < 2^32) as 32-bit words."""
    out = torch.empty((rows, cols), dtype=torch.int32, device="cuda")
    if p <= 1 << 31:
        out.random_(0, p, generator=g)
        return out
    wide = torch.empty((rows, cols), dtype=torch.int64, device="cuda").random_(0, p, generator=g)
    return torch.where(wide >= 1 << 31, wide - (1 << 32), wide).to(torch.int32)


def _uniform64(g, rows: int, cols: int, p: int) -> torch.Tensor:
    return torch.empty((rows, cols), dtype=torch.int64, device="cuda").random_(0, p, generator=g)


def _factors(g, m: int, n: int, r: int, p: int):
    """Factors m x r and r x n whose product has rank r: uniform ones, which have full rank but for a
    chance of about 1/p; over the small fields triangular ones with rows and columns in random order."""
    L, R = _uniform(g, m, r, p), _uniform(g, r, n, p)
    if p < 1 << 15:
        one = torch.eye(r, dtype=torch.int32, device="cuda")
        L[:r] = torch.tril(L[:r], -1) + one
        R[:, :r] = torch.triu(R[:, :r], 1) + one
        L = L[torch.randperm(m, generator=g, device="cuda")]
        R = R[:, torch.randperm(n, generator=g, device="cuda")].contiguous()
    return L, R


def _planted(n: int, ell: int, k: int, zeros: int, seed: int):
    """U D V mod ell^k and the exponents of D: U, V products of 64 elementary row
    operations with multipliers in [-5, 5], D = diag(ell^e), e geometric(1/2) on
    [0, k) but for `zeros` zeros on the diagonal (the construction of
    ``gen.planted_udv`` applied in place, with the rank given by the case)."""
    q = ell ** k
    r = np.random.default_rng(int(seed))
    e = (r.geometric(0.5, n) - 1) % k
    e[r.choice(n, zeros, replace=False)] = k
    ops = []
    for _ in range(128):
        i, j = r.choice(n, 2, replace=False)
        ops.append((int(i), int(j), int(r.integers(-5, 6))))
    M = np.eye(n, dtype=np.int64)
    for i, j, c in ops[:64]:
        M[i] = (M[i] + c * M[j]) % q
    M = M * np.array([pow(ell, int(x)) if x < k else 0 for x in e], dtype=np.int64)[:, None] % q
    for i, j, c in ops[64:]:
        M[i] = (M[i] + c * M[j]) % q
    return M.astype(np.uint32), e


def _zeros(case) -> int:
    """Smith: the truncated distribution's expected number of zeros; Howell: none (every column has a pivot)."""
    return case["n"] >> case["k"] if case["op"] == "smith" else 0


def _stream(case, seed: int) -> DeviceStream:
    """The job stream's shapes, families and moduli, its entries from `seed`."""
    s = DeviceStream(case["count"], salt=case["salt"])
    key = gen.seed_for(case["count"], 0, case["salt"] + 1, int(seed))
    s.specs = [(t, p, fam, (int(sd) ^ key) & gen.MASK64) for t, p, fam, sd in s.specs]
    return s


def prepare(case, seed):
    op = case["op"]
    eng = _engine(own=op == "jobs")
    st = {"eng": eng, "op": op, "case": case}
    if op in ("gemm", "gemm_u64", "gemv"):
        g, p, fill = _gen(seed), case["p"], _uniform64 if op == "gemm_u64" else _uniform
        m, k, n = case["m"], case["k"], case.get("n", 1)
        st["A"], st["B"] = fill(g, m, k, p), fill(g, k, n, p)
        st["C"] = fill(g, m, n, p)
        if case["acc"] != "set":
            st["C0"] = st["C"].clone()
    elif op == "rref":
        g, p, m, n, r = _gen(seed), case["p"], case["m"], case["n"], case["rank"]
        L, R = _factors(g, m, n, r, p)
        st["A"] = torch.empty((m, n), dtype=torch.int32, device="cuda")
        eng.gemm_dev(p, L, R, st["A"])
        torch.cuda.synchronize()  # L and R are dropped here
        st["W"] = torch.empty_like(st["A"])
    elif op in ("howell", "smith"):
        st["A"], _ = _planted(case["n"], case["ell"], case["k"], _zeros(case), seed)
    else:
        s = _stream(case, seed)
        eng.gen_jobs_dev(s.specs)
        eng.sync()
        st["stream"], st["jobs"] = s, s.jobs
    return st


def run(st):
    eng, op, c = st["eng"], st["op"], st["case"]
    if op in ("gemm", "gemm_u64", "gemv"):
        if "C0" in st:  # the accumulator as the pass finds it
            st["C"].copy_(st["C0"])
        if op == "gemm":
            eng.gemm_dev(c["p"], st["A"], st["B"], st["C"], OPS[c["acc"]])
        elif op == "gemm_u64":
            eng.gemm_u64_dev(c["p"], st["A"], st["B"], st["C"], OPS[c["acc"]])
        else:
            eng.gemv_dev(c["p"], st["A"], st["B"], st["C"], OPS[c["acc"]])
        return st["C"]
    if op == "rref":  # in place, so on a copy
        st["W"].copy_(st["A"])
        piv = eng.rref_dev(c["p"], st["W"])
        return st["W"], piv
    if op == "howell":
        return eng.howell(c["ell"], c["k"], st["A"])
    if op == "smith":
        return eng.smith(c["ell"], c["k"], st["A"])
    return eng.batch_gemm_rank_dev(st["jobs"])


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    """Bytes: every input read once, every output written once.  flops: two per modular multiply-add of
    the classical algorithm (a product: mnk; an echelon form of rank r: LU mnr - r^2 (m + n)/2 + r^3/3 and
    r^2 (n - r)/2 for the reduction above the pivots; a Howell or Smith form: n^3/3)."""
    op = case["op"]
    if op in ("gemm", "gemm_u64", "gemv"):
        m, k, n = case["m"], case["k"], case.get("n", 1)
        w = 8 if op == "gemm_u64" else 4
        return {"bytes": w * (m * k + k * n + (m * n if case["acc"] == "set" else 2 * m * n)), "flops": 2.0 * m * n * k}
    if op == "rref":
        m, n, r = case["m"], case["n"], case["rank"]
        lu = m * n * r - r * r * (m + n) / 2 + r ** 3 / 3
        return {"bytes": 8 * m * n, "flops": 2.0 * (lu + r * r * (n - r) / 2)}
    if op in ("howell", "smith"):
        n = case["n"]
        return {"bytes": (8 if op == "howell" else 4) * n * n, "flops": 2.0 * n ** 3 / 3}
    s = gen.job_stream(case["count"], case["salt"])[0].astype(np.float64)
    return {"bytes": 8 * float((s ** 2).sum()), "flops": 2.0 * float((4 * s ** 3 / 3).sum())}


# ---- the same results in plain torch -------------------------------------------------------------
def _product(A: torch.Tensor, B: torch.Tensor, p: int) -> torch.Tensor:
    """A B mod p of words below 2^32, by 16-bit halves in exact float64 sums (k 2^32 < 2^53)."""
    def halves(t):
        t = t.to(torch.int64) & 0xFFFFFFFF
        return (t >> 16).double(), (t & 0xFFFF).double()

    (ah, al), (bh, bl) = halves(A), halves(B)

    def mod(x):
        return x.to(torch.int64) % p

    hi, mid, lo = mod(ah @ bh), mod(ah @ bl) + mod(al @ bh), mod(al @ bl)
    return (((hi * 65536 % p + mid) % p) * 65536 + lo) % p


def exact(case, seed):
    op = case["op"]
    if op == "smith":  # the planted valuations below k
        _, e = _planted(case["n"], case["ell"], case["k"], _zeros(case), seed)
        return np.sort(e[e < case["k"]]).astype(np.uint32)
    if op not in ("gemm", "gemv"):
        return None
    st = prepare(case, seed)
    p = case["p"]
    prod = _product(st["A"], st["B"], p)
    if case["acc"] != "set":
        c0 = st["C0"].to(torch.int64) & 0xFFFFFFFF
        prod = (c0 + prod) % p if case["acc"] == "add" else (c0 - prod) % p
    return torch.where(prod >= 1 << 31, prod - (1 << 32), prod).to(torch.int32)

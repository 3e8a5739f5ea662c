"""The products' reduction by one 32-bit multiply-high, in Python integers: its constants for the sums that the
limb products, the limb split and the residue system's last sum reach, at multiples of p and at the bounds."""
import random

import pytest

M32 = (1 << 32) - 1
MODULI = [2, 3, 128, 255, 256, 257, 511, 512, 65535, 65536, 65537, 131071, 131073, (1 << 24) - 1, 1 << 24,
          (1 << 24) + 43, (1 << 25) + 1, (1 << 31) - 1, 1 << 31, (1 << 31) + 11, (1 << 32) - 17, (1 << 32) - 5, M32]


def _limbs(p):
    return 1 if p <= 256 else 2 if p <= 65536 else 3 if p <= 1 << 24 else 4


def _bounds(p):
    L = _limbs(p)
    chunk = ((1 << 31) - 1) // (L * 255 * 255) // 128 * 128
    for k in (1, 64, 129, 1000, chunk):
        yield sum((L * 255 * 255 * k) << (8 * j) for j in range(L))  # a product's chunk of K
    yield 256 << (8 * L)                                             # the split of B
    if L == 4:
        yield 22 * 255 * 255 * 0x01010101 + (22 << 32)               # the residue system's last sum


def _reduce(s, p, bound):
    """(constants as make_epi_bound gives them, the result as epi_reduce_u64 does)."""
    b, sb = p.bit_length(), bound.bit_length()
    sh1 = max(0, sb - 32)
    sh2 = b - 1 - sh1
    assert 0 <= sh1 <= 31 and 0 <= sh2 <= 31
    M = min(M32, (1 << (31 + b)) // p)
    hi = s >> sh1
    assert hi <= M32
    q = ((hi * M) >> 32) >> sh2
    x = s - q * p
    assert x >= 0
    if p < 1 << 31 and sh1 <= b - 2:  # one word: min(x, x - p)
        assert x < 2 * p
        return min(x, (x - p) & M32)
    assert x < 3 * p
    assert p < 1 << 31 or x < 2 * p
    x -= p if x >= p else 0
    return min(x, (x - p) & M32)


@pytest.mark.parametrize("p", MODULI)
def test_sums_up_to_their_bounds(p):
    rnd = random.Random(p)
    for bound in _bounds(p):
        top = bound // p
        tests = {0, 1, bound, bound - 1}
        for k in [1, 2, top, max(0, top - 1)] + [rnd.randint(0, top) for _ in range(300)]:
            tests |= {k * p - 1, k * p, k * p + 1, k * p + p - 1}
        for e in range(bound.bit_length()):
            tests |= {(1 << e) - 1, 1 << e}
        for s in tests:
            if 0 <= s <= bound:
                assert _reduce(s, p, bound) == s % p, (s, bound)

"""The tensor-core setup's arithmetic (csrc/setup_tc.cu), emulated in exact integers on the CPU: balanced
base-256 digits of a word against those of the position residues in byte planes, one biased fp32 sum per
plane, and neighbouring planes combined straight from the sums' bits.  Integers: equal, no tolerance."""
import random

import pytest

DIGITS, BIAS, TBIAS = 225, 0x4B400000, 0x8B400000


def balanced(v, n):
    """n digits of -128..127 (the last takes the carry), as bytes of v + 0x8080.. less 128."""
    v += sum(128 << 8 * i for i in range(n - 1))
    return [((v >> 8 * i) & 255) - 128 for i in range(n - 1)] + [v >> 8 * (n - 1)]


def planes(w, p, n):
    """n digits of w in [0, p), or of w - p where w passes what they hold."""
    top = int("7F" * n, 16)
    v = (w - p if n == 4 and w > top else w) + int("80" * n, 16)
    assert 0 <= v < 1 << 8 * n
    return [((v >> 8 * i) & 255) - 128 for i in range(n)]


@pytest.mark.parametrize("p,n", [(3, 4), (65537, 4), (1000000007, 4), (2**31 - 1, 4), (2**31 + 11, 8),
                                 (2**40 + 15, 8), (6148914691236517189, 8)])
def test_word_sums_are_exact_and_congruent(p, n):
    rng = random.Random(p)
    w = [planes((1 << 8 * b + 32) % p, p, n) for b in range(DIGITS)]
    const = sum(TBIAS << 16 * j for j in range(n // 2))
    off = planes(-const % p, p, n)
    words = [0, 1, 2**1792 - 1, int("80" * 224, 16), int("7F" * 224, 16), 2**1791] + [rng.getrandbits(1792) for _ in range(20)]
    for Z in words:
        z = balanced(Z, DIGITS)
        assert all(-128 <= d <= 127 for d in z) and z[-1] in (0, 1)
        bits = []
        for a in range(n):
            s, lo, hi = off[a], off[a], off[a]
            for d, wb in zip(z, w):
                s += d * wb[a]
                lo, hi = min(lo, s), max(hi, s)
            assert -2**22 <= lo and hi < 2**22   # every partial sum on the bias of 1.5 2^23 is exact
            bits.append(BIAS + s)
        t = [(bits[2 * j] + 256 * bits[2 * j + 1]) % 2**32 for j in range(n // 2)]
        assert all(v == bits[2 * j] - BIAS + 256 * (bits[2 * j + 1] - BIAS) + TBIAS for j, v in enumerate(t))
        T = sum(v << 16 * j for j, v in enumerate(t))
        assert T % p == (Z << 32) % p and T < (2**48 if n == 4 else 2**80)

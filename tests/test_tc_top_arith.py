"""The arithmetic of the tensor-core kernels' canonical class 64 (candidates from 2^64/3 on, in csrc/setup_tc.cu and
csrc/walk_tc.cu), emulated on the CPU: digits of a residue that passes what eight of them hold, sums that wrap past
2^64 before they are reduced, and the walk's test with its residue cut to 32 bits and rounded in fp32 as the kernel
does.  Integers: equal, no tolerance."""
import random

import numpy as np
import pytest

from tests import test_tc_digits as td
from tests import test_walk_tc_arith as wa

PRIMES = [2**62 + 135, 2**64 // 3 + 4, 2**63 + 29, 3 * 2**62 + 125, 2**64 - 59, 2**64 - 1]   # (odd is enough)
M64 = 2**64 - 1


def reduced(u, t, p):
    """u = (T + m p) / 2^32, summed modulo 2^64 with its last addend t: less p where it wrapped or passes p."""
    u &= M64
    return (u - p) & M64 if u < t or u >= p else u


@pytest.mark.parametrize("p", PRIMES)
def test_setup_words(p):
    rng = random.Random(p)

    def planes(w):
        v = ((w - p if w > 0x7F7F7F7F7F7F7F7F else w) + 0x8080808080808080) & M64
        d = [((v >> 8 * i) & 255) - 128 for i in range(8)]
        assert (sum(x << 8 * i for i, x in enumerate(d)) - w) % p == 0
        return d

    w = [planes((1 << 8 * b + 32) % p) for b in range(td.DIGITS)]
    off = planes(-sum(td.TBIAS << 16 * j for j in range(4)) % p)
    assert all(-128 <= x <= 127 for r in w + [off] for x in r)
    q = pow(p, -1, 2**64)
    words = [0, 1, 2**1792 - 1, int("80" * 224, 16), int("7F" * 224, 16)] + [rng.getrandbits(1792) for _ in range(40)]
    for Z in words:
        z = td.balanced(Z, td.DIGITS)
        s = [off[a] + sum(d * wb[a] for d, wb in zip(z, w)) for a in range(8)]
        assert all(-2**22 <= x < 2**22 for x in s)
        t = [(td.BIAS + s[2 * j] + 256 * (td.BIAS + s[2 * j + 1])) % 2**32 for j in range(4)]
        T = sum(v << 16 * j for j, v in enumerate(t))
        assert T % p == (Z << 32) % p and T < 2**80
        L, H = t[0] + (t[1] << 16), t[2] + (t[3] << 16)
        tw0, mh = L & wa.M32, (L >> 32) + H
        mm = -tw0 * q & wa.M32
        lo = mm * (p & wa.M32)
        assert (tw0 + lo) & wa.M32 == 0
        u = mm * (p >> 32) + (lo >> 32) + (tw0 != 0) + mh
        assert u == (T + mm * p) >> 32
        u = reduced(u, mh, p)
        assert u < p and u == Z % p


@pytest.mark.parametrize("bits", [46, 48])
@pytest.mark.parametrize("p", PRIMES)
def test_sums_that_wrap(p, bits):
    """The reductions' last addend, below 2^48 (setup) or 2^46 (walk), on multiples of p near 2^32 p."""
    wrapped = passed = 0
    for m in [0, 1, 2**31, wa.M32 - 1, wa.M32]:
        tw0 = -m * p & wa.M32
        first = (m * p + tw0) >> 32
        for t in [0, 1, 2**32, 2**bits - 1, p - first - 1, p - first, 2**64 - first]:
            if not 0 <= t < 1 << bits:
                continue
            wrapped += first + t > M64
            passed += first + t >= p
            assert reduced(first + t, t, p) == (first + t) % p
    assert passed and (wrapped or p < 2**64 - 2**bits)


@pytest.mark.parametrize("top,KD,nb", [(202000, 47, 16), (12900000, 63, 16), (2**31 - 1, 63, 12)])
@pytest.mark.parametrize("p", PRIMES)
def test_block_product_advances_the_residue(p, top, KD, nb):
    rng = random.Random(p + top)
    w = [(pow(2, 96, p) << 6 * b) % p for b in range(KD)]
    pinv = pow(p, -1, 2**64)
    r = plain = rng.randrange(1, p)
    r = r * 2**64 % p
    for _ in range(50):
        W = 1
        for _ in range(nb):
            W *= rng.randrange(top - top // 50, top + 1)
        d = [(W >> 6 * b) & 63 for b in range(KD)]
        S = [sum(x * ((y >> o) & ((1 << z) - 1)) for x, y in zip(d, w))
             for o, z in zip((0, 11, 22, 32, 43, 54), (11, 11, 10) * 2)]
        assert all(x < 2**23 for x in S)
        L, H = (S[k] + (S[k + 1] << 11) + (S[k + 2] << 22) for k in (0, 3))
        m = -(L & wa.M32) * pinv & wa.M32
        c = m * (p & wa.M32) + (L & wa.M32)
        t = H + (L >> 32)
        u = m * (p >> 32) + (c >> 32) + t
        assert c < 2**64 and t < 2**46 and u == (L + (H << 32) + m * p) >> 32
        u = reduced(u, t, p)
        assert u < p
        r = r * u * pow(2, -64, p) % p
        plain = plain * W % p
        assert r == plain * 2**64 % p


def fraction16(r, p):
    """A as the kernel forms it: fp32 of the residue's top word, one fused multiply-add, 16 bits of the result."""
    scale = np.float32(4194304.0) / np.float32(np.ldexp(np.float64(np.float32(np.uint64(p))), -32))
    # (24 x 24 bits and an addend of 2^23: exact in a double, then the one rounding)
    f = np.float32(np.float64(np.float32(np.uint32(r >> 32))) * np.float64(scale) + 12582912.0)
    return (int(f.view(np.uint32)) >> 6) & 0xFFFF


@pytest.mark.parametrize("top,KD,nb", [(130, 47, 16), (202000, 47, 16), (202001, 63, 16), (12900000, 63, 16),
                                       (2**31 - 1, 63, 12)])
@pytest.mark.parametrize("p", PRIMES)
def test_hits_pass_the_window(p, top, KD, nb):
    rng = random.Random(p ^ top)
    blocks = []
    for _ in range(40):
        n0 = rng.randrange(max(101, top - 5000), top - nb + 1) if top > 200 else 101
        N = [1]
        for i in reversed(range(nb)):
            N.append(N[-1] * (n0 + i))
        blocks.append(N)
    half = max(wa.window(N[:nb], KD) for N in blocks)
    hi, lo = wa.planes_f(p, 2**64, KD, half)
    for N in blocks:
        for j in range(nb):
            y = wa.mid16(N[j], hi, lo, KD)
            for r in (N[j] % p, -N[j] % p):
                assert wa.passes(y, fraction16(r * 2**64 % p, p), half)


@pytest.mark.parametrize("p", PRIMES)
def test_the_fraction_is_within_its_bound(p):
    """A is 16 bits, cut, of a fraction that is off by less than 0.045 of them."""
    rng = random.Random(p)
    for r in [0, 1, 2**32 - 1, 2**32, p - 1, p - 2**32, p // 2, p // 3] + [rng.randrange(p) for _ in range(3000)]:
        exact = r * 65536 / p   # (a double: far below the bound)
        a = fraction16(r, p)
        off = min((a - exact) % 65536, (exact - a) % 65536)
        d = (exact - a + 32768) % 65536 - 32768   # in [-0.045, 1.045]
        assert -0.045 <= d <= 1.045 and off <= 1.045

"""The tensor-core walk's arithmetic (csrc/walk_tc.cu), emulated in exact integers on the CPU.

A block's tests compare fractions: with r the residue at the block's end and N_j the product of its last j
multipliers, N_j = +-r (mod p) means frac(N_j R / p) = +-frac(r R / p).  The emulation forms the words' digits,
the candidate's planes, the sums and the 16-bit test as the kernel does, and checks that every true hit
passes the window, that random pairs pass about as often as the window is wide, that every sum keeps its
place in the fp32 mantissa, and that the block product advances the residue exactly.
"""
import random

import pytest

BIAS_F, BIAS_E = 0x4B400000, 0x4B000000
M32, M64 = 2**32 - 1, 2**64 - 1


def planes_f(p, R, KD, half):
    """Test planes: 24 bits of frac(2^(6b) R / p) from its 32-bit expansion, rounded, as two 12-bit digits."""
    w = R % p
    e = []
    pinv = pow(p, -1, 2**32)
    for _ in range(14):
        w2 = (w << 32) % p
        q = (-w2 * pinv) & M32
        assert q == (w << 32) // p
        e.append(q)
        w = w2
    hi, lo = [], []
    for b in range(KD):
        bit = 6 * b
        t = ((e[bit // 32] << 32 | e[bit // 32 + 1]) >> (32 - bit % 32)) & M32
        f = (t + 0x80) >> 8
        lo.append(((f + 2048) & 4095) - 2048)
        hi.append((((f + 2048) >> 12) + 2048 & 4095) - 2048)
        assert (hi[-1] * 4096 + lo[-1] - f) % 2**24 == 0
    # the last digit, 1 in every test word: takes off what the biases leave, adds half + 1 units of 2^-16
    hi[-1], lo[-1] = -1024, 256 * (half + 1)
    return hi, lo


def balanced(n, KD):
    v = n + sum(32 << 6 * b for b in range(KD - 1))
    assert v < 1 << 6 * (KD - 1)
    return [((v >> 6 * b) & 63) - 32 for b in range(KD - 1)] + [1]


def mid16(n, hi, lo, KD):
    d = balanced(n, KD)
    s = [sum(x * y for x, y in zip(d, f)) for f in (hi, lo)]
    assert all(abs(x) < 2**22 for x in s)
    x = ((BIAS_F + s[0]) * 4096 + BIAS_F + s[1]) & M32
    return (x >> 8) & 0xFFFF


def passes(y, A, half):
    return min((y + (A ^ 0xFFFF)) & 0xFFFF, (y + A) & 0xFFFF) <= 2 * half


def window(words, KD):
    """The half window of a table: f_b off by up to 0.504 units of 2^-24, A by 0.045 of 2^-16."""
    digits = max(sum(abs(d) for d in balanced(n, KD)[:-1]) for n in words)
    return int(digits * (0.504 / 256) + 0.045) + 1


@pytest.mark.parametrize("top,KD,nb", [(130, 47, 16), (202000, 47, 16), (202001, 63, 16), (12900000, 63, 16),
                                       (2**31 - 1, 63, 12)])
@pytest.mark.parametrize("p,R", [(65537, 2**32), (2**31 - 1, 2**32), (1000000007, 2**32), (2**31 + 11, 2**64),
                                 (2**40 + 15, 2**64), (6148914691236517189, 2**64)])
def test_hits_pass_the_window(p, R, top, KD, nb):
    rng = random.Random(p ^ top)
    blocks = []
    for _ in range(40):
        n0 = rng.randrange(max(101, top - 5000), top - nb + 1) if top > 200 else 101
        N = [1]
        for i in reversed(range(nb)):
            N.append(N[-1] * (n0 + i))
        assert N[nb] < 1 << 6 * KD
        blocks.append(N)
    by_chance = 0
    half = max(window(N[:nb], KD) for N in blocks)
    assert half <= 4
    hi, lo = planes_f(p, R, KD, half)
    for N in blocks:
        for j in range(nb):
            y = mid16(N[j], hi, lo, KD)
            for r in (N[j] % p, -N[j] % p):
                for lift in (0, 1 if R == 2**64 else -1):   # the kept residue: [0, 2p), or (-p, p)
                    x = r * R % p + lift * p
                    scale = 4194304 if R == 2**32 else 2097152
                    for err in (-0.8, 0, 0.8):   # the fp32 product, in units of its last place kept
                        f = round(x * scale / p + err)
                        A = (f >> (6 if R == 2**32 else 5)) & 0xFFFF
                        assert passes(y, A, half)
            by_chance += passes(y, rng.randrange(65536), half)
    if p > 2**20 and top > 200:
        assert by_chance <= 3 + 40 * nb * 2 * (2 * half + 1) / 65536 * 4


@pytest.mark.parametrize("top,KD,nb", [(202000, 47, 16), (12900000, 63, 16), (2**31 - 1, 63, 12)])
@pytest.mark.parametrize("p", [3, 65537, 2**31 - 1, 1000000007, 2**31 + 11, 2**40 + 15, 6148914691236517189])
def test_block_product_advances_the_residue(p, top, KD, nb):
    rng = random.Random(p + top)
    narrow = p < 2**31
    R = 2**32 if narrow else 2**64
    w = [(pow(2, 64 if narrow else 96, p) << 6 * b) % p for b in range(KD)]
    offs = (0, 11, 22) if narrow else (0, 11, 22, 32, 43, 54)
    size = (11, 11, 10) * 2
    pinv = pow(p, -1, 2**32)
    r = rng.randrange(1, p) * R % p
    plain = r
    for _ in range(50):
        W = 1
        for _ in range(nb):
            W *= rng.randrange(top - top // 50, top + 1)
        d = [(W >> 6 * b) & 63 for b in range(KD)]
        assert W >> 6 * KD == 0
        S = [sum(x * ((y >> o) & ((1 << z) - 1)) for x, y in zip(d, w)) for o, z in zip(offs, size)]
        assert all(x < 2**23 for x in S)
        T = sum(s << o for s, o in zip(S, offs))
        assert T < p << 12 and T % p == W * w[0] % p
        plain = plain * W % p
        if narrow:
            m = (T * pinv) & M32
            m -= (m >> 31) << 32
            u = (T >> 32) - ((m * p) >> 32)
            assert abs(u) <= p / 2 + 2**11
            t = r * u
            m = ((t & M32) * pinv) & M32
            m -= (m >> 31) << 32
            r = (t >> 32) - ((m * p) >> 32)
            assert abs(r) < p
        else:
            u = (T + (-T * pinv & M32) * p) >> 32
            assert u < p + 2**43
            c = (r * (u & M32) + (-(r * (u & M32)) * pinv & M32) * p) >> 32
            c += r * (u >> 32)
            r = (c + (-c * pinv & M32) * p) >> 32
            assert 0 <= r < 2 * p
        assert r % p == plain

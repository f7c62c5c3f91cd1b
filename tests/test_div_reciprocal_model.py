"""CPU model of block division's reciprocal (divtc.cuh, dt_recip): Newton's iteration
with the kernel's left-out columns, from the reciprocal of the divisor's top two
limbs.  Its error stays below the bound derived there for every divisor -- the
worst for a one-limb start are divisors whose top limb is just above 2^63 and
whose next limb is all ones -- and the quotient block it estimates differs from
the true one by at most one, and seldom."""
import random

import pytest

B = 1 << 64


def _limbs(x, n):
    return [(x >> (64 * i)) & (B - 1) for i in range(n)]


def _int(x):
    return sum(v << (64 * i) for i, v in enumerate(x))


def _recip(V, LW):
    v, p = _limbs(V, LW) + [0], 1
    y = (B ** 3 - 1) // (v[LW - 1] * B + v[LW - 2]) - B
    while p < LW:
        top, Y = v[LW - 2 * p:], _limbs(y, p)

        def columns(X):         # column p - 1 and up of X Y
            return sum((X[p - 1 + t - i] * Y[i]) << (64 * t) for t in range(p + 2) for i in range(p)) >> 64

        S = (columns(top) + _int(top[:p + 1])) % B ** (p + 1)
        pos = S >> (64 * (p + 1) - 1) == 0
        E = S if pos else B ** (p + 1) - S
        D = columns(_limbs(E, p + 1) + [0] * p) + E
        y = max(0, min((y << (64 * p)) + (-D if pos else D), B ** (2 * p) - 1))
        p *= 2
    return y


def _divisors(rng, LW):
    bits = 64 * LW
    for top in [0, 1, 2, 3, 0x2a4, (1 << 20) + 1, (1 << 62) - 1, (1 << 63) - 1] + [rng.getrandbits(rng.randrange(1, 64))
                                                                                 for _ in range(24)]:
        for second in (B - 1, B - 2, 0, rng.getrandbits(64)):
            for below in (0, 1, (1 << (bits - 128)) - 1, rng.getrandbits(bits - 128), rng.getrandbits(64)):
                yield (1 << 63 | top) << (bits - 64) | second << (bits - 128) | below


@pytest.mark.parametrize("LW,bound", [(32, 1 << 29), (64, 1 << 57)])
def test_error_of_any_divisor(LW, bound):
    rng = random.Random(11)
    for V in _divisors(rng, LW):
        assert abs(_recip(V, LW) - ((B ** (2 * LW) - 1) // V - B ** LW)) < bound, hex(V >> (64 * LW - 128))


def test_derived_bound():
    """The recurrence of dt_recip's comment."""
    lo, hi = 0, 1                                   # bounds of eta, the residual in units of the last limb
    for p in (1, 2, 4, 8, 16, 32):
        neg = lo < 0
        lo, hi = -(p + 2) - (p if neg else 0), max(lo * lo, hi * hi) + p
        if p == 16:
            assert 2 * max(-lo, hi) + 1 < 1 << 29
    assert 2 * max(-lo, hi) + 1 < 1 << 57


@pytest.mark.parametrize("LW", [32, 64])
def test_quotient_blocks(LW):
    rng, off, seen = random.Random(13), 0, 0
    KB = LW - 1
    for V in _divisors(rng, LW):
        inv = _limbs(_recip(V, LW), LW)
        for _ in range(2 if LW == 32 else 1):
            q = rng.getrandbits(64 * KB)
            W = q * V + rng.randrange(V)            # a window of 2 LW - 1 limbs over V
            wt = _limbs(W >> (64 * (LW - 1)), LW)
            cols = sum((wt[a] * inv[c - a]) << (64 * (c - KB)) for c in range(KB, 2 * LW - 1)
                       for a in range(max(0, c - KB), min(c, KB) + 1))
            est = min(((cols >> 64) + _int(wt)) >> 64, B ** KB - 1)
            assert abs(est - q) <= 1
            off += est != q
            seen += 1
    assert off <= seen // 20

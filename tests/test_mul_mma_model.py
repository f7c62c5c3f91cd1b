"""CPU model of the warp matrix product (mulmma.cuh): balanced digits with their
carry digit, a's padded image and b's two pair images, the fragments each lane
reads from them and the pairing of fragments into tiles give the product; every
index stays inside its image, and the sums between two moves to integers stay
within 2^24."""
import random

import numpy as np
import pytest

B = 1 << 64
HALF = 0x8080808080808080


def _digits(x, limbs):
    t = x + HALF * ((B ** limbs - 1) // (B - 1))
    return [v - 128 for v in (t % B ** limbs).to_bytes(8 * limbs, "little")], t >> (64 * limbs)


def _model(LT, full, a, b, out_limbs):
    N, U = 128 * LT, 2 * LT if full else LT
    da, ca = _digits(a, 16 * LT)
    db, cb = _digits(b, 16 * LT)
    A = np.zeros(N + 128 + 144, np.int64)
    A[128:128 + N] = da
    A[128 + N] = ca
    be, bo = np.zeros((N // 2 + 16, 2), np.int64), np.zeros((N // 2 + 16, 2), np.int64)
    for k in range(N // 2):
        bo[8 + k] = db[2 * k + 1], db[2 * k]
        be[8 + k] = db[2 * k], db[2 * k - 1] if k else 0
    be[8 + N // 2] = cb, db[N - 1]
    bo[8 + N // 2] = 0, cb
    i, k = np.arange(16)[:, None], np.arange(16)[None, :]

    def F(s):
        at = 128 + 16 * s + 8 * i + k
        assert at.min() >= 0 and at.max() < A.size
        return A[at]

    def G(g):
        m = np.zeros((16, 8), np.int64)
        for lane in range(32):
            q, t = lane >> 2, lane & 3
            for reg in (0, 1):
                at = 8 + (q >> 1) - t + 8 * g - 4 * reg
                assert 0 <= at < N // 2 + 16
                m[2 * t + 8 * reg, q], m[2 * t + 1 + 8 * reg, q] = (bo if q & 1 else be)[at]
        return m

    C, total = np.zeros((U, 16, 8), np.int64), np.zeros((U, 16, 8), np.int64)
    for r in range(8):
        bs = {w: G(8 * w - r) for w in range(1, LT + 1)}
        for v in range(-1, LT):
            for w in bs:
                if v + w < U:
                    C[v + w] += F(r + 8 * v) @ bs[w]
        if full and r == 0:
            for w in range(1, LT):
                C[LT + w] += F(8 * LT) @ bs[w]
        if LT > 8 and r == 3:
            assert abs(C).max() <= 1 << 24
            total, C = total + C, C * 0
    for v in range(LT + 1 if full else LT):
        C[v] += F(8 * v) @ G(0)
    assert abs(C).max() <= 1 << 24
    total += C
    val = sum(int(x) << (8 * d) for d, x in enumerate(total.reshape(-1)))
    assert val % B ** out_limbs == a * b % B ** out_limbs


@pytest.mark.parametrize("full,LTs", [(True, range(1, 11)), (False, range(1, 17))])
def test_products(full, LTs):
    rng = random.Random(3)
    for LT in LTs:
        for L in {16 * LT - 15, 16 * LT - 1, 16 * LT}:
            pats = [rng.getrandbits(64 * L), (1 << (64 * L)) - 1, int.from_bytes(b"\x80" * (8 * L), "little"),
                    int.from_bytes(b"\x7f" * (8 * L), "little")]
            for a in pats:
                _model(LT, full, a, pats[rng.randrange(4)], 2 * L if full else L)

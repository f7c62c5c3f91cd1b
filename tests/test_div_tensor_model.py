"""CPU model of block division on the tensor cores (divtc.cuh): its scaling and
block count, the Newton reciprocal (lane sums and left-out columns as in the
kernel), the estimate, the digit images, descriptors and column order, the
signed carries between segments and the corrections give exact quotients and
remainders; addresses stay inside their buffers, column sums below 2^22 or 2^23.  With
`off` the estimates are moved by one either way, so that both corrections run."""
import random

import numpy as np
import pytest

B = 1 << 64


def _limbs(x, n):
    return [(x >> (64 * i)) & (B - 1) for i in range(n)]


def _int(x):
    return sum(v << (64 * i) for i, v in enumerate(x))


def _recip(V, LW):
    """Kernel's dt_recip: about floor((B^2LW - 1) / V) - B^LW."""
    v, y = _limbs(V, LW) + [0], [0] * LW
    y[-1] = (B * B - 1) // v[LW - 1] - B
    p = 1
    while p < LW:
        v2, Y = v[LW - 2 * p:], y[LW - p:]

        def column_sum(X):
            return sum((X[p - 1 + t - i] * Y[i]) << (64 * t) for t in range(p + 2) for i in range(p))

        S = ((column_sum(v2) >> 64) + _int(v2[:p + 1])) % B ** (p + 1)
        pos = S >> (64 * (p + 1) - 1) == 0
        E = S if pos else B ** (p + 1) - S
        D = (column_sum(_limbs(E, p + 1) + [0] * p) >> 64) + E
        Yn = (_int(Y) << (64 * p)) + (-D if pos else D)
        y[LW - 2 * p:] = _limbs(max(0, min(Yn, B ** (2 * p) - 1)), 2 * p)
        p *= 2
    return _int(y)


@pytest.mark.parametrize("LW,bound", [(32, 1 << 30), (64, 1 << 56)])
def test_reciprocal(LW, bound):
    rng, bits = random.Random(7), 64 * LW
    for i in range(600 if LW == 32 else 200):
        V = rng.getrandbits(bits) | 1 << (bits - 1)
        if i % 5 == 1:
            V = (1 << bits) - 1 - rng.getrandbits(rng.randrange(1, bits - 1))
        elif i % 5 == 2:
            V = (1 << (bits - 1)) + rng.getrandbits(rng.randrange(1, bits - 1))
        elif i % 5 == 3:
            V = (1 << (bits - 1)) if i % 2 else (1 << bits) - 1
        assert abs(_recip(V, LW) - (((1 << (2 * bits)) - 1) // V - (1 << bits))) < bound


def _divide(P, H, LW, u, v, MU, rng, off):
    KB = LW - 1
    Q, QT, T0 = P // 8, P // 8 // H, -8 * LW
    steps = (P - T0) // 16
    CM, kmin = Q + 2 * steps - 1, -((-T0 + P - 1) // P)
    R = (128 - kmin + 6) // 8 * 8 + 1
    qlo, qhi = 2 * steps - LW, Q + 1
    K = -(-v.bit_length() // 64)
    assert R >= 128 - kmin and K <= 128 * Q - KB - 2
    s, Kp = 64 * K - v.bit_length(), max(K, LW)
    z = Kp - K
    V, U = (v << s) << (64 * z), (u << s) << (64 * z)
    nb = (MU + 1 - K + KB - 1) // KB
    assert nb * KB + Kp <= MU + 2 * LW and U < B ** (nb * KB + Kp)
    win, lim = _limbs(U, nb * KB + Kp), Kp + KB
    inv = _limbs(_recip(V >> (64 * (Kp - LW)), LW), LW) + [0] * LW
    half = 0x8080808080808080
    ob = (V + half * ((B ** (Kp + 1) - 1) // (B - 1))).to_bytes(8 * (Kp + 1), "little")
    A = np.zeros(R * Q * 8, np.int64)
    for x in range(Kp + 1):
        at = ((x % Q) * R + x // Q - kmin) * 8
        A[at:at + 8] = [c - 128 for c in ob[8 * x:8 * x + 8]]
    i, kk, n = np.arange(128), np.arange(16), np.arange(P)
    quot = [0] * MU
    for blk in range(nb - 1, -1, -1):
        w0 = blk * KB
        wt = win[w0 + Kp - 1:w0 + Kp + KB]
        cols = sum((wt[a] * inv[c - a]) << (64 * (c - KB)) for c in range(KB, 2 * LW - 1) for a in range(LW))
        cols -= sum(wt[a] * inv[KB - a] for a in range(LW)) % B
        q = min(((cols >> 64) + _int(wt)) >> 64, B ** KB - 1)
        if off:
            q = max(0, min(B ** KB - 1, q + rng.choice([0, 1, -1])))
        raw = [0x80] * (8 * qlo) + list((q + half * ((B ** LW - 1) // (B - 1))).to_bytes(8 * LW, "little")) + [0x80] * (8 * qhi)
        st = np.zeros(CM * 64, np.int64)
        for x in range(CM):
            for j0 in range(8):
                at = 8 * (qlo + Q - 2 - T0 // 8 - x) + j0 + 1
                assert at >= 0 and at // 4 * 4 + 12 <= len(raw)
                st[x * 64 + j0 * 8:x * 64 + j0 * 8 + 8] = [c - 128 for c in raw[at:at + 8][::-1]]
        acc = np.zeros((128, P), np.int64)
        for k in range(steps):
            t = T0 + 16 * k
            sa = t // P - kmin + t % P // 8 * R
            assert 0 <= sa and sa + R + 127 < R * Q and 2 * k + Q < CM
            acc += (A[(sa + i[:, None] + (kk // 8)[None, :] * R) * 8 + (kk % 8)[None, :]]
                    @ st[2 * k * 64 + ((n // 8) * 64 + n % 8 * 8)[:, None] + (kk // 8 * 64 + kk % 8)[None, :]].T)
        assert abs(acc).max() <= (1 << 22 if LW == 32 else 1 << 23)
        val, cs = [], []
        for sg in range(128 * H):
            c, x = (0 if sg == 0 else -(1 << 30)), 0
            for k in range(QT):
                limb = sg % H * QT + k
                col = acc[sg // H][8 * (Q - 1 - limb):8 * (Q - limb)]
                at = QT * sg + k
                t = (win[w0 + at] if at < lim else 0) + c - sum(int(a) << (8 * e) for e, a in enumerate(col))
                x += (t % B) << (64 * k)
                c = t >> 64
            assert -(1 << 30) <= c < 1 << 30
            val.append(x)
            cs.append(c)
        carry, res = 0, []
        for sg in range(128 * H):
            x = val[sg] + (0 if sg == 0 else cs[sg - 1] + (1 << 30)) + carry
            carry = x >> (64 * QT)
            assert carry in (0, 1)
            res += _limbs(x, QT)
        neg = cs[-1] + carry < 0
        win[w0:w0 + lim] = res[:lim]
        W = _int(res[:lim])
        if neg:
            assert res[Kp] >> 63
            W -= B ** lim
        else:
            assert W < B ** (Kp + 1)
        if not neg and win[w0 + Kp] == 0 and win[w0 + Kp - 1] < V >> (64 * (Kp - 1)):
            assert W < V
        fixes = 0
        while not 0 <= W < V:
            W, q = (W + V, q - 1) if W < 0 else (W - V, q + 1)
            fixes += 1
        assert fixes <= 3
        win[w0:w0 + lim] = _limbs(W, lim)
        for t, x in enumerate(_limbs(q, KB)):
            if w0 + t < MU:
                quot[w0 + t] = x
            else:
                assert x == 0
    return _int(quot), (_int(win[:Kp]) >> (64 * z)) >> s


@pytest.mark.parametrize("P,H,LW,sizes", [(16, 1, 32, (1, 2, 31, 32, 33, 100, 223)), (32, 1, 32, (224, 479)),
                                          (48, 1, 32, (735,)), (64, 1, 32, (991,)), (80, 2, 64, (1, 63, 64, 1024, 1215)),
                                          (128, 2, 32, (2015,)), (128, 2, 64, (1983,))])
def test_division(P, H, LW, sizes):
    rng = random.Random(P)
    for K in sizes:
        for rep in range(6 if K < 300 else 2):
            bits = 64 * K
            v = [rng.getrandbits(bits) | 1, (1 << bits) - 1, 1 << (bits - 1), rng.getrandbits(bits - 9) | 1 << (bits - 10),
                 int.from_bytes(b"\x80" * (8 * K), "little"), (1 << (bits - 1)) + rng.getrandbits(bits // 2)][rep]
            MU = K + rng.choice([0, 1, LW - 2, LW - 1, 2 * LW - 2])
            u = [rng.getrandbits(64 * MU), (1 << (64 * MU)) - 1, v * rng.getrandbits(64 * (MU - K) + 1) - 1][rep % 3]
            u = max(0, min(u, (1 << (64 * MU)) - 1))
            for off in (False, True):
                assert _divide(P, H, LW, u, v, MU, rng, off) == divmod(u, v), (P, K, MU, rep, off)

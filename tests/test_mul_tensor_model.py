"""CPU model of the tensor-core product's index arithmetic (multc.cuh): A's and
B's shared-memory images, the descriptors' addresses into them, the ranges of
blocks and the accumulator's column order give the digit convolution, every
address stays inside its buffer and every block's sums stay below 2^23."""
import random

import numpy as np
import pytest


def _krange(D, tau):
    return max(-D, -(128 * tau + 127)), min(0, D - 1 - 128 * tau)


def _model(P, L, out, rng):
    Q, RB = P // 8, 128 // P
    KB = RB * P
    CM = Q + KB // 8 - 1
    D, tiles = -(-L // Q), -(-out // (128 * Q))
    spans = []
    for tau in range(tiles):
        lo, hi = _krange(D, tau)
        assert hi >= lo
        nblk = (hi - lo + RB) // RB
        spans.append((128 * tau + lo, 128 * tau + 127 + lo + nblk * RB - 1))
    rho0 = min(s for s, _ in spans)
    R = max(e for _, e in spans) - rho0 + 1
    R += (9 - R % 8) % 8
    ones = rng.random() < 0.3
    a = [255 if ones else rng.randrange(256) for _ in range(8 * L)]
    b = [255 if ones else rng.randrange(256) for _ in range(8 * L)]
    A = np.zeros(R * Q * 8, np.int64)
    for x in range(L):
        at = (x % Q * R + x // Q - rho0) * 8
        assert 0 <= at <= A.size - 8
        A[at:at + 8] = a[8 * x:8 * x + 8]
    PAD, top = 16, 2 * Q + 1
    braw = [0] * (8 * PAD) + b + [0] * (8 * top)
    C = np.zeros(tiles * 128 * P, np.int64)
    i, kk, n = np.arange(128), np.arange(16), np.arange(P)
    for tau in range(tiles):
        lo, hi = _krange(D, tau)
        acc = np.zeros((128, P), np.int64)
        for k0 in range(lo, hi + 1, RB):
            st = np.zeros(CM * 64, np.int64)
            for x in range(CM):
                w = Q - 1 - Q * k0 - x
                for j0 in range(8):
                    at = 8 * (PAD + w - 1) + j0 + 1          # bytes j0 - 7 .. j0 of limb w
                    assert 0 <= at and at + 11 < len(braw)   # three aligned words from at's word on
                    st[x * 64 + j0 * 8:x * 64 + j0 * 8 + 8] = braw[at:at + 8][::-1]
            blk = np.zeros((128, P), np.int64)
            for s in range(KB // 16):
                sa = 128 * tau + k0 - rho0 + 16 * s // P + (16 * s % P // 8) * R
                assert sa >= 0 and sa + R + 127 < R * Q
                assert 2 * s + (Q - 1) + 1 < CM
                Am = A[(sa + i[:, None] + (kk // 8)[None, :] * R) * 8 + (kk % 8)[None, :]]
                Bm = st[2 * s * 64 + ((n // 8) * 64 + (n % 8) * 8)[:, None] + (kk // 8 * 64 + kk % 8)[None, :]]
                blk += Am @ Bm.T
            assert blk.max() < 1 << 23
            acc += blk
        assert acc.max() < 1 << 32
        for col in range(P):
            C[(128 * tau + i) * P + 8 * (Q - 1 - col // 8) + col % 8] = acc[:, col]
    ref = np.convolve(a, b)
    ref = np.concatenate([ref, np.zeros(max(0, C.size - ref.size), np.int64)])
    assert (C[:8 * out] == ref[:8 * out]).all()


@pytest.mark.parametrize("P", [16, 32, 64, 96, 128])
def test_layouts_give_the_convolution(P):
    rng = random.Random(P)
    for L in (1, 15, 16, 17, 33, 64, 65, 128, 257, 512):
        for out in (L, 2 * L):
            if out <= 128 * (P // 8) * 3:
                _model(P, L, out, rng)

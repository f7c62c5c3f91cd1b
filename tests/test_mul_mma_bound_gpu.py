"""Products on the warp's matrix instruction where its f32 sums are largest: operands
whose balanced digits are all -128 (B^L - 0x8080..80), some raised to -127 so that
a sum past 2^24 could not be held, at both ends of every size class and around the
sizes where a truncated product's columns pass 1024 products in a half."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operands(seed, n, m, w):
    rng = random.Random(seed)
    size = m * w // 8
    low = (1 << (8 * size)) - int.from_bytes(b"\x80" * size, "little")

    def value(i):
        x = low
        for _ in range((0, 1, 1, 2, 5, 40)[i % 6]):     # distinct places: a digit is at most -127
            k = rng.randrange(size)
            if x >> (8 * k) & 255 == low >> (8 * k) & 255:
                x += 1 << (8 * k)
        return x

    return [value(i) for i in range(n)], [value(i // 6) for i in range(n)]


def _dev(vals, m, w):
    import torch

    raw = b"".join(v.to_bytes(m * w // 8, "little") for v in vals)
    return torch.from_numpy(np.frombuffer(raw, np.int64 if w == 64 else np.int32).reshape(len(vals), m).copy()).cuda()


def _check(B, m, w, full):
    n = 160                                             # more than one an SM
    a, b = _operands(m * 2 + w, n, m, w)
    bits = m * w
    r = (B.mulfull if full else B.mul)(_dev(a, m, w), _dev(b, m, w))
    got = [int.from_bytes(row.tobytes(), "little") for row in r.cpu().numpy()]
    want = [x * y if full else x * y % (1 << bits) for x, y in zip(a, b)]
    assert got == want, (m, w, full)


@pytest.mark.parametrize("m", sorted({L for k in range(1, 17) for L in (16 * k - 15, 16 * k)} | {248, 249, 250, 251, 255}))
def test_largest_sums(bigint, m):
    for full in (False, True):
        _check(bigint, m, 64, full)
        _check(bigint, max(1, 2 * m - 1), 32, full)     # an odd word count

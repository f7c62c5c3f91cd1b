"""Block division where its reciprocal and its digit sums are at their limits, against
Python integers: divisors whose top limb is just above 2^63 and whose next limb is
all ones (the worst start of Newton's iteration), divisors whose balanced digits
are all -128 (B^K - 0x8080..80), quotients of -128 digits, and dividends that are a
multiple of the divisor, or one below the next."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(vals, m, w):
    import torch

    raw = b"".join(v.to_bytes(m * w // 8, "little") for v in vals)
    return torch.from_numpy(np.frombuffer(raw, np.int64 if w == 64 else np.int32).reshape(len(vals), m).copy()).cuda()


def _ints(t):
    return [int.from_bytes(row.tobytes(), "little") for row in t.cpu().numpy()]


def _low(size):
    return (1 << (8 * size)) - int.from_bytes(b"\x80" * size, "little")


def _instances(seed, mu, mv, n, w):
    rng = random.Random(seed)
    bu, bv = mu * w, mv * w
    us, vs = [], []
    for i in range(n):
        top = (1 << 63) | (0, 1, 0x2a4, 3, rng.getrandbits(40), (1 << 62) + 1)[i % 6]
        v = top << (bv - 64) | (((1 << 64) - 1) << (bv - 128)) | rng.getrandbits((1, 64, bv - 128)[i % 3])
        if i % 4 == 3:
            v = _low(mv * w // 8)
            if i % 8 == 3:
                v += 1 << (8 * rng.randrange(mv * w // 8 - 1))
        most = ((1 << bu) - 1) // v
        q = _low((bu - bv) // 8) if i % 5 == 4 and bu > bv else rng.randrange(most)
        us.append(min((1 << bu) - 1, q * v + (0, v - 1, rng.randrange(v))[i % 3]))
        vs.append(v)
    return us, vs


def _check(B, mu, mv, n, w):
    us, vs = _instances(mu * 37 + mv, mu, mv, n, w)
    q, r, st = B.div(_dev(us, mu, w), _dev(vs, mv, w))
    for i, (u, v, a, b, s) in enumerate(zip(us, vs, _ints(q), _ints(r), st.cpu().tolist())):
        assert (a, b, s) == (*divmod(u, v), 0), (mu, mv, w, i)


@pytest.mark.parametrize("mu,mv,n", [(64, 40, 24), (130, 65, 24), (512, 256, 200), (958, 479, 24), (1470, 735, 24),
                                     (1982, 991, 24), (2048, 1024, 170), (2430, 1215, 24), (2494, 1247, 24),
                                     (3966, 1983, 24), (3000, 1500, 160), (4030, 2015, 24)])
def test_against_integers(bigint, mu, mv, n):
    _check(bigint, mu, mv, n, 64)
    _check(bigint, 2 * mu - 1, 2 * mv - 1, 24, 32)

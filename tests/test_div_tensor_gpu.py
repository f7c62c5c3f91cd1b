"""Division in blocks of 31 or 63 quotient limbs on the tensor cores against Python
integers: both sides of every accumulator width, one to many quotient blocks,
divisors with leading zero limbs (down to one limb), powers of two, all ones,
bytes of 0x80 (the largest balanced digits), dividends just below a multiple of
the divisor, zero divisors, one instance and more instances than CTAs, odd u32
word counts."""
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


def _instances(seed, mu, mv, n, w):
    rng = random.Random(seed)
    bu, bv = mu * w, mv * w
    us, vs = [], []
    for i in range(n):
        v = rng.getrandbits(bv) | 1 << (bv - 1)
        k = i % 10
        if k == 1:
            v >>= rng.randrange(0, w)
        elif k == 2:
            v >>= rng.randrange(0, bv)
        elif k == 3:
            v = (1 << bv) - 1
        elif k == 4:
            v = 1 << rng.randrange(bv)
        elif k == 5:
            v = int.from_bytes(b"\x80" * (bv // 8), "little")
        elif k == 6:
            v = (1 << (bv - 1)) + rng.getrandbits(bv // 3)
        elif k == 7 and i > 10:
            v = 0
        u = rng.getrandbits(bu)
        if k in (3, 8):
            u = (1 << bu) - 1
        elif k in (6, 9):
            u = max(0, min((1 << bu) - 1, v * ((1 << (bu - bv)) + rng.getrandbits(max(1, bu - bv))) - 1))
        elif i % 20 == 11:
            u = max(0, min((1 << bu) - 1, v - 1))
        us.append(u)
        vs.append(v)
    return us, vs


def _check(B, mu, mv, n, w):
    us, vs = _instances(mu * 31 + mv, mu, mv, n, w)
    q, r, st = B.div(_dev(us, mu, w), _dev(vs, mv, w))
    for i, (u, v, a, b, s) in enumerate(zip(us, vs, _ints(q), _ints(r), st.cpu().tolist())):
        want = (0, 0, 1) if v == 0 else (*divmod(u, v), 0)
        assert (a, b, s) == want, (mu, mv, w, i)


@pytest.mark.parametrize("mu,mv,n", [
    (64, 40, 12), (130, 65, 12), (129, 66, 700), (200, 130, 24), (446, 223, 24), (447, 224, 24), (512, 256, 320),
    (958, 479, 12), (960, 480, 12), (1470, 735, 12), (1472, 736, 12), (1982, 991, 12), (1984, 992, 12),
    (2048, 1024, 170), (2430, 1215, 12), (2432, 1216, 12), (2494, 1247, 160), (3966, 1983, 12), (3968, 1984, 12),
    (4030, 2015, 12), (3000, 1500, 160), (1055, 1024, 12), (1054, 1024, 12),
    (2030, 2010, 12), (8192, 1000, 4), (8192, 2015, 4), (8192, 65, 4)])
def test_against_integers(bigint, mu, mv, n):
    _check(bigint, mu, mv, n, 64)
    _check(bigint, 2 * mu - 1, 2 * mv - 1, min(n, 12), 32)


def test_status_may_be_left_out(bigint):
    import torch

    B = bigint
    us, vs = _instances(5, 300, 150, 4, 64)
    u, v = _dev(us, 300, 64), _dev(vs, 150, 64)
    q, r = torch.empty_like(u), torch.empty_like(v)
    st = B.lib().bi_div_u64(u.data_ptr(), v.data_ptr(), q.data_ptr(), r.data_ptr(), None, 300, 150, 4, None)
    torch.cuda.synchronize()
    assert st == 0
    assert [(a, b) for a, b in zip(_ints(q), _ints(r))] == [divmod(a, b) for a, b in zip(us, vs)]

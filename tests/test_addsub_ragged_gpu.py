"""Sums and differences of sizes that are no multiple of 64 bytes in aligned
buffers, against Python's integers: one chunk and its edges, one CTA's largest
instance and the next, fewer and more tiles than CTAs, a last tile that is not
full, operands that carry or borrow all the way, equal and neighbouring
operands, results in place, and the limbs beside the output."""
import numpy as np
import pytest

from bigint_gb300.workloads import uniform_limbs

pytestmark = pytest.mark.gpu


def _ints(x):
    return [int.from_bytes(row.tobytes(), "little") for row in x]


def _operands(seed, n, m, dtype):
    a = uniform_limbs(seed, n, m, dtype)
    b = uniform_limbs(seed + 1, n, m, dtype)
    ones = np.iinfo(dtype).max
    for k in range(n):
        kind = k % 8
        if kind == 0:
            a[k], b[k] = ones, 0
            b[k, 0] = 1                                          # a carry through every limb
        elif kind == 1:
            a[k], b[k] = 0, 0
            b[k, 0] = 1                                          # and a borrow
        elif kind == 2:
            b[k] = a[k]
        elif kind == 3:
            b[k] = a[k]
            b[k, m - 1] ^= dtype(1)
        elif kind == 4:
            a[k] = ones
            b[k] = ones
    return a, b


@pytest.mark.parametrize("bits,m,ns", [
    (64, 5, (1, 51, 60000)), (64, 7, (255, 257)), (64, 9, (3, 50001)), (64, 13, (1000,)), (64, 15, (17, 20001)),
    (64, 255, (1, 3001)), (64, 1785, (500,)), (64, 1792, (2,)), (64, 1793, (1, 320)), (64, 3583, (160,)), (64, 3585, (3,)),
    (32, 7, (1, 60001)), (32, 14, (500,)), (32, 15, (255, 257, 40001)), (32, 17, (30001,)), (32, 31, (1, 7777)),
    (32, 33, (1001,)), (32, 333, (1, 2001)), (32, 3839, (600,)), (32, 3841, (1, 310)), (32, 7679, (153,)), (32, 7681, (3,))])
def test_sizes(bigint, bits, m, ns):
    import torch

    B = bigint
    dtype = np.uint64 if bits == 64 else np.uint32
    mod = 1 << (bits * m)
    for n in ns:
        a, b = _operands(7000 + m, n, m, dtype)
        x, y = _ints(a), _ints(b)
        da, db = B.to_device(a), B.to_device(b)
        buf = torch.full((n * m + 16,), 77, dtype=da.dtype, device="cuda")
        r = buf[8:8 + n * m].view(n, m)                          # 16-byte aligned, no more
        sign = torch.full((n + 1,), 9, dtype=torch.uint8, device="cuda")
        diff, sums = [abs(p - q) for p, q in zip(x, y)], [(p + q) % mod for p, q in zip(x, y)]
        neg = [int(p < q) for p, q in zip(x, y)]
        B.sub(da, db, r, sign[:n])
        assert _ints(B.to_host(r, dtype)) == diff and sign.cpu().tolist() == neg + [9], (m, n)
        B.add(da, db, r)
        assert _ints(B.to_host(r, dtype)) == sums, (m, n)
        assert bool((buf[:8] == 77).all()) and bool((buf[8 + n * m:] == 77).all())
        r.copy_(da)
        B.sub(r, db, r, sign[:n])                                # over its first operand
        assert _ints(B.to_host(r, dtype)) == diff and sign.cpu().tolist() == neg + [9], (m, n)
        r.copy_(db)
        B.add(da, r, r)                                          # over its second
        assert _ints(B.to_host(r, dtype)) == sums, (m, n)

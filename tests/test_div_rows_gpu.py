"""Divisions of one thread each whose rows pass through shared memory, and those
that read them in place, against Python's integers: warps that are not full, odd
and even limb and word counts, the longest rows and the next, more instances than
the rows' limit, divisors with zero high limbs, zero divisors, quotient limbs at
and one below their estimate, and the limbs beside the outputs."""
import numpy as np
import pytest

from bigint_gb300.workloads import uniform_limbs

pytestmark = pytest.mark.gpu


def _ints(x):
    return [int.from_bytes(row.tobytes(), "little") for row in x]


def _operands(seed, n, mu, mv, dtype):
    u = uniform_limbs(seed, n, mu, dtype)
    v = uniform_limbs(seed + 1, n, mv, dtype)
    ones = np.iinfo(dtype).max
    for k in range(0, n, 7):
        v[k, mv - 1 - (k // 7) % mv:] = 0                        # shorter, zero at times
    for k in range(3, n, 11):
        u[k] = ones
        v[k] = [ones, 0, 1][k % 3]
        v[k, mv - 1] = [ones, 1, ones // 2 + 1][k % 3]
    for k in range(5, n, 13):
        v[k] = ones
        u[k, mu - mv:] = ones
        u[k, mu - mv] -= dtype(1)
    return u, v


@pytest.mark.parametrize("bits,mu,mv,ns", [
    (64, 1, 1, (1, 31, 33)), (64, 4, 2, (63, 65, 60000)), (64, 9, 3, (100,)), (64, 16, 8, (32, 1000, 60000)),
    (64, 15, 7, (64, 60000)), (64, 25, 12, (127, 60000)), (64, 56, 16, (7400,)), (64, 57, 16, (7400,)),
    (64, 48, 8, (60000,)), (64, 49, 8, (60000,)), (64, 71, 1, (33,)), (64, 72, 1, (33,)),
    (32, 2, 1, (1, 64)), (32, 7, 5, (60000,)), (32, 16, 7, (33, 60000)), (32, 31, 15, (95, 60000)), (32, 32, 16, (60000,)),
    (32, 155, 31, (7400,)), (32, 156, 32, (7400,)), (32, 158, 32, (7400,)), (32, 143, 3, (40,)), (32, 141, 2, (40,))])
def test_rows(bigint, bits, mu, mv, ns):
    import torch

    B = bigint
    dtype = np.uint64 if bits == 64 else np.uint32
    for n in ns:
        u, v = _operands(8000 + mu + mv, n, mu, mv, dtype)
        du, dv = B.to_device(u), B.to_device(v)
        qb = torch.full((n * mu + 2,), 77, dtype=du.dtype, device="cuda")
        rb = torch.full((n * mv + 2,), 77, dtype=du.dtype, device="cuda")
        q, r = qb[1:-1].view(n, mu), rb[1:-1].view(n, mv)
        status = torch.full((n + 1,), 9, dtype=torch.uint8, device="cuda")
        B.div(du, dv, q, r, status[:n])
        code = status.cpu().tolist()
        assert code[n] == 9
        rows = zip(_ints(u), _ints(v), _ints(B.to_host(q, dtype)), _ints(B.to_host(r, dtype)), code)
        for k, (x, y, a, b, c) in enumerate(rows):
            assert (a, b, c) == ((*divmod(x, y), 0) if y else (0, 0, 1)), (mu, mv, n, k)
        for buf in (qb, rb):
            assert int(buf[0]) == 77 and int(buf[-1]) == 77

"""Products on the warp's matrix instruction (one warp an instance) against the
oracle: every size class and both sides of its edges, full and truncated, 64-bit
limbs and odd word counts, buffers off a 16-byte boundary, operands whose bytes
are all 255, 0x80 and 0x7f (carries out of the balanced digits, the largest
column sums), zeros, neighbours of the output, and batches of one warp and of
more than the grid."""
import numpy as np
import pytest

from bigint_gb300.workloads import uniform_limbs

pytestmark = pytest.mark.gpu


def _operands(seed, n, m, dtype):
    a = uniform_limbs(seed, n, m, dtype)
    b = uniform_limbs(seed + 1, n, m, dtype)
    one = np.iinfo(dtype).max // 255                             # 0x0101..01
    for k, (x, y) in enumerate([(255, 255), (0x80, 0x80), (0x7F, 0x80), (0x80, 255), (0, 255), (0x7F, 0x7F)]):
        if k < n - 1:
            a[k], b[k] = dtype(one * x), dtype(one * y)
    return a, b


def _check(B, oracle, a, b, full, shift=0):
    import torch

    n, m = a.shape
    k = 2 * m if full else m

    def place(x):
        buf = torch.full((x.size + 2 + shift,), 77, dtype=B.to_device(x[:1]).dtype, device="cuda")
        t = buf[1 + shift:1 + shift + x.size].view(x.shape)
        t.copy_(B.to_device(x))
        return buf, t

    _, da = place(a)
    _, db = place(b)
    buf, r = place(np.zeros((n, k), a.dtype))
    (B.mulfull if full else B.mul)(da, db, out=r)
    ref = oracle.mulfull(a, b) if full else oracle.mul(a, b)
    assert (B.to_host(r, a.dtype) == ref).all(), (m, a.dtype, full, shift)
    assert bool((buf[:1 + shift] == 77).all()) and int(buf[-1]) == 77


# 160 instances: more than one an SM, few enough for the small sizes to come here too
@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("m", [8, 9, 15, 16, 17, 24, 25, 31, 32, 33, 48, 49, 64, 65, 80, 81, 96, 97, 112, 113, 128, 129,
                               144, 145, 160, 161, 175, 177, 192, 193, 208, 209, 224, 225, 240, 241, 255, 256])
def test_size_classes(bigint, oracle, m, full):
    a, b = _operands(4000 + m, 160, m, np.uint64)
    _check(bigint, oracle, a, b, full, shift=1)                  # 16-byte aligned
    _check(bigint, oracle, a[:9], b[:9], full)                   # 8 bytes off
    w = 2 * m - 1
    a, b = _operands(4100 + m, 160, w, np.uint32)
    _check(bigint, oracle, a, b, full)
    if m in (16, 33, 64, 130):
        a, b = _operands(4200 + m, 20, w - 1, np.uint32)         # an even count: limbs if 8-byte aligned
        _check(bigint, oracle, a, b, full)
        _check(bigint, oracle, a, b, full, shift=1)


@pytest.mark.parametrize("m,n", [(20, 1), (20, 9000), (30, 5000), (64, 1), (64, 20000), (100, 9000), (150, 5000)])
def test_batch_sizes(bigint, oracle, m, n):
    a, b = _operands(4300 + m, n, m, np.uint64)
    for full in (True, False):
        _check(bigint, oracle, a, b, full, shift=1)

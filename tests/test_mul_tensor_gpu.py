"""Products on the tensor cores against the oracle: both sides of every
accumulator width and tile count, operands whose digits are all 255 (the
largest column sums), zeros, one instance and more instances than CTAs, odd
u32 word counts, and neighbours of the output left alone."""
import numpy as np
import pytest

from bigint_gb300.workloads import uniform_limbs

pytestmark = pytest.mark.gpu


def _operands(seed, n, m, dtype):
    a = uniform_limbs(seed, n, m, dtype)
    b = uniform_limbs(seed + 1, n, m, dtype)
    top = np.iinfo(dtype).max
    a[0] = top
    b[0] = top
    if n > 2:
        a[1] = 0
        b[2] = 0
        b[2, -1] = top
    return a, b


def _check(B, oracle, a, b):
    import torch

    n, m = a.shape
    da, db = B.to_device(a), B.to_device(b)
    for full in (True, False):
        k = 2 * m if full else m
        buf = torch.full((n * k + 2,), 77, dtype=da.dtype, device="cuda")
        r = buf[1:-1].view(n, k)
        (B.mulfull if full else B.mul)(da, db, out=r)
        ref = oracle.mulfull(a, b) if full else oracle.mul(a, b)
        assert (B.to_host(r, a.dtype) == ref).all(), (m, a.dtype, full)
        assert int(buf[0]) == 77 and int(buf[-1]) == 77


# full products of 2 m limbs: widths change above 256, 512, 1024 and 1536
# product limbs, a second tile starts above 2048, a third above 4096
@pytest.mark.parametrize("m", [33, 64, 127, 128, 129, 160, 208, 255, 256, 257, 512, 513, 768, 769, 1000, 1024, 1025,
                               1536, 1537, 2048, 2049, 3000, 4096])
@pytest.mark.parametrize("dtype", [np.uint64, np.uint32])
def test_widths_and_tiles(bigint, oracle, m, dtype):
    n = 3 if m > 600 else 5
    if dtype == np.uint32:
        m = 2 * m - 1                      # an odd word count: the top limb is half empty
    _check(bigint, oracle, *_operands(9000 + m, n, m, dtype))


@pytest.mark.parametrize("m,n", [(48, 1), (64, 1216), (250, 700), (512, 400), (1024, 160)])
def test_one_instance_and_many(bigint, oracle, m, n):
    _check(bigint, oracle, *_operands(9100 + m, n, m, np.uint64))


def test_same_in_a_graph(bigint, oracle):
    import torch

    B = bigint
    a, b = _operands(9200, 40, 300, np.uint64)
    da, db = B.to_device(a), B.to_device(b)
    r = torch.zeros((40, 600), dtype=torch.int64, device="cuda")
    B.mulfull(da, db, out=r)
    r.zero_()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        B.mulfull(da, db, out=r)
    g.replay()
    assert (B.to_host(r, np.uint64) == oracle.mulfull(a, b)).all()

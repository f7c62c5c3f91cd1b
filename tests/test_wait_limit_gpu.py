"""A device-side wait that runs out: the kernel ends by itself, writes no result, and
the failure reaches the host -- bi_wait_status and every later call answer
BI_ETIMEDOUT until it is cleared, and then calls are exact again.  The wait is made
to run out by a barrier that expects an arrival which nothing sends."""
import subprocess
import sys

import numpy as np
import pytest

from bigint_gb300.workloads import uniform_limbs

pytestmark = pytest.mark.gpu

TIMED_OUT = 4


@pytest.fixture
def waits(bigint):
    assert bigint.wait_status() == 0
    yield bigint
    import torch

    torch.cuda.synchronize()
    bigint.wait_status(clear=True)


def _held(B, kind, a, b, r, status, m, n):
    import torch

    assert B.lib().bi_probe_held_wait(kind, a.data_ptr(), b.data_ptr(), r.data_ptr(), status.data_ptr(), m, n,
                                      torch.cuda.current_stream().cuda_stream) == 0, B.lib().bi_last_error()
    torch.cuda.synchronize()                       # the kernel ended and the context is usable


def _refused(B, call):
    with pytest.raises(B.BigIntError) as e:
        call()
    assert e.value.status == TIMED_OUT


def _check_reported(B, oracle):
    a, b = uniform_limbs(1, 40, 200), uniform_limbs(2, 40, 200)
    da, db = B.to_device(a), B.to_device(b)
    assert B.wait_status() == TIMED_OUT
    for call in (B.add, B.sub, B.mul, B.mulfull, B.div, B.cmp):
        _refused(B, lambda: call(da, db))
    _refused(B, lambda: B.add_chain(da, db, 3))
    _refused(B, lambda: B.mul_chain(da, db, 3))
    _refused(B, lambda: B.mul_autotune(da, db))
    _refused(B, lambda: B.host_mulfull(a, b))
    assert B.wait_status() == TIMED_OUT            # until it is cleared
    assert B.wait_status(clear=True) == TIMED_OUT and B.wait_status() == 0
    assert (B.to_host(B.mulfull(da, db), np.uint64) == oracle.mulfull(a, b)).all()
    assert B.wait_status() == 0


@pytest.mark.parametrize("m,n", [(5, 2), (128, 24)])
def test_products(waits, oracle, m, n):
    import torch

    B = waits
    a, b = B.to_device(uniform_limbs(3, n, m)), B.to_device(uniform_limbs(4, n, m))
    r = torch.full((n, 2 * m), 77, dtype=torch.int64, device="cuda")
    _held(B, 0, a, b, r, torch.zeros(n, dtype=torch.uint8, device="cuda"), m, n)
    assert bool((r == 77).all())
    _check_reported(B, oracle)


@pytest.mark.parametrize("m,n", [(7, 2), (125, 64)])
def test_differences(waits, oracle, m, n):
    """One tile, and five on one CTA with the next one's copies under way."""
    import torch

    B = waits
    a, b = B.to_device(uniform_limbs(3, n, m)), B.to_device(uniform_limbs(4, n, m))
    r = torch.full((n, m), 77, dtype=torch.int64, device="cuda")
    sign = torch.full((n,), 77, dtype=torch.uint8, device="cuda")
    _held(B, 1, a, b, r, sign, m, n)
    assert bool((r == 77).all()) and bool((sign == 77).all())
    _check_reported(B, oracle)
    assert (B.to_host(B.sub(a, b)[0], np.uint64) == oracle.sub(B.to_host(a, np.uint64), B.to_host(b, np.uint64))[0]).all()


@pytest.mark.parametrize("m,n", [(40, 2), (128, 24)])
def test_divisions(waits, oracle, m, n):
    """One division and twelve a CTA: status 2 for all, also those after the one that waited."""
    import torch

    B = waits
    a, b = B.to_device(uniform_limbs(3, n, 2 * m)), B.to_device(uniform_limbs(4, n, m))
    r = torch.full((3 * n * m,), 77, dtype=torch.int64, device="cuda")
    status = torch.full((n,), 77, dtype=torch.uint8, device="cuda")
    _held(B, 2, a, b, r, status, m, n)
    assert bool((status == 2).all())
    _check_reported(B, oracle)
    q, rem, st = B.div(a, b)
    wq, wr, ws = oracle.div(B.to_host(a, np.uint64), B.to_host(b, np.uint64))
    assert (B.to_host(q, np.uint64) == wq).all() and (B.to_host(rem, np.uint64) == wr).all() and not st.any()


def test_plan_is_refused(waits):
    import torch

    B = waits
    d, arena, out_limbs, nflags = B.workloads.uneven_batch(n=60, seed=5, max_bits=32768)
    din = B.to_device(arena)
    out = torch.zeros(out_limbs, dtype=torch.int64, device="cuda")
    fl = torch.zeros(nflags, dtype=torch.uint8, device="cuda")
    plan = B.Plan(d, din.numel(), out_limbs, nflags)
    a = B.to_device(uniform_limbs(6, 2, 8))
    _held(B, 0, a, a, torch.zeros((2, 16), dtype=torch.int64, device="cuda"), fl, 8, 2)
    _refused(B, lambda: plan.execute(din, out, fl))
    _refused(B, lambda: plan.autotune(din, out, fl))
    torch.cuda.synchronize()
    assert not bool(out.any())                     # nothing was launched
    B.wait_status(clear=True)
    plan.execute(din, out, fl)
    torch.cuda.synchronize()
    assert bool(out.any())
    plan.close()


def test_first_call_inside_a_capture(bigint):
    """The word that reports a wait is set up by the first call that needs it,
    which may be one that is being captured."""
    code = """
import sys; sys.path.insert(0, sys.argv[1])
import torch, bigint_gb300 as B
a = torch.randint(-2**62, 2**62, (64, 300), dtype=torch.int64, device="cuda")
r = torch.zeros((64, 600), dtype=torch.int64, device="cuda")
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    B.mulfull(a, a, out=r)
g.replay()
torch.cuda.synchronize()
x = int.from_bytes(a[5].cpu().numpy().tobytes(), "little")
assert int.from_bytes(r[5].cpu().numpy().tobytes(), "little") == x * x
assert B.wait_status() == 0
"""
    import os

    path = os.path.dirname(os.path.dirname(os.path.abspath(bigint.__file__)))
    p = subprocess.run([sys.executable, "-c", code, path], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]

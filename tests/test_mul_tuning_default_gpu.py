"""What the multiply autotuner reports for the tensor cores is no CTA tiling: replayed
through mul_set_tuning it leaves the library's own choice in force, also after a
tiling was pinned by hand; (1, 1) still pins that tiling."""
import numpy as np
import pytest

from bigint_gb300.workloads import uniform_limbs

pytestmark = pytest.mark.gpu


def _us(fn, reps=5):
    import torch

    for _ in range(3):
        fn()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(reps):
        fn()
    e1.record()
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / reps * 1e3


@pytest.mark.parametrize("m,dtype", [(1024, np.uint64), (2048, np.uint32)])
def test_replayed_choice_keeps_the_tensor_cores(bigint, oracle, m, dtype):
    B = bigint
    a, b = uniform_limbs(1, 600, m, dtype), uniform_limbs(2, 600, m, dtype)
    da, db = B.to_device(a), B.to_device(b)
    try:
        chosen = B.mul_autotune(da, db, full=True, reps=3)
        assert chosen == (B.MUL_DEFAULT, 1)        # four times as fast as any tiling here
        own = _us(lambda: B.mulfull(da, db))
        B.mul_set_tuning(m, dtype, True, 1, 1)
        pinned = _us(lambda: B.mulfull(da, db))
        B.mul_set_tuning(m, dtype, True, *chosen)
        replayed = _us(lambda: B.mulfull(da, db))
        assert pinned > 2 * own and pinned > 2 * replayed
        k = 8
        assert (B.to_host(B.mulfull(da, db), dtype)[:k] == oracle.mulfull(a[:k], b[:k])).all()
    finally:
        B.mul_set_tuning(m, dtype, True, 0)

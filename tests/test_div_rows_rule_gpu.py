"""Both sides of the lines between divisions whose rows pass through shared memory and
those that read them in place, by quotient length and batch size, against Python's
integers."""
import numpy as np
import pytest

from test_div_rows_gpu import _ints, _operands

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,mv,qls,ns", [
    (64, 1, (1, 7, 8), (1, 1000)), (64, 4, (7, 8, 23, 24), (33, 24400)), (64, 7, (7, 8), (300,)), (64, 8, (7, 8), (500, 9800)),
    (32, 5, (7, 8), (300,)), (32, 14, (4, 5), (300, 24400)), (32, 8, (4, 5), (300,)), (32, 16, (1, 2), (12000,))])
def test_lines(bigint, bits, mv, qls, ns):
    B = bigint
    dtype = np.uint64 if bits == 64 else np.uint32
    for ql in qls:
        mu = mv + ql - 1 if bits == 64 else 2 * ((mv + 1) // 2 + ql - 1)
        for n in ns:
            u, v = _operands(8200 + mu + mv, n, mu, mv, dtype)
            q, r, st = B.div(B.to_device(u), B.to_device(v))
            rows = zip(_ints(u), _ints(v), _ints(B.to_host(q, dtype)), _ints(B.to_host(r, dtype)), st.cpu().tolist())
            for k, (x, y, a, b, c) in enumerate(rows):
                assert (a, b, c) == ((*divmod(x, y), 0) if y else (0, 0, 1)), (mu, mv, n, k)

"""How many digit products meet in one f32 sum of the warp matrix product
(mulmma.cuh).  A product of balanced digits is at most 2^14, so the sums between
two moves to integers are exact whatever their order as long as at most 1024 of
them meet in a column.  Counted tile by tile in the kernel's order, for every
size class, with every digit of both operands and their carry digits present."""
import numpy as np
import pytest


def _counts(LT, full):
    """Products in each column's sum, for each part between two moves to integers."""
    N, U = 128 * LT, 2 * LT if full else LT
    A = np.zeros(N + 272, np.int64)
    A[128:128 + N + 1] = 1                      # the digits and the carry digit, zeros around them
    Bd = np.zeros(N + 64, np.int64)
    Bd[32:32 + N + 1] = 1
    i, k, j = np.arange(16)[:, None], np.arange(16)[None, :], np.arange(8)[None, :]

    def F(s):
        return A[128 + 16 * s + 8 * i + k]

    def G(g):
        at = 32 + 16 * g + j - np.arange(16)[:, None]
        return Bd[at]

    parts, C = [], np.zeros((U, 16, 8), np.int64)
    for v in range(LT + 1 if full else LT):     # residue 0, g = 0, comes first
        C[v] += F(8 * v) @ G(0)
    for r in range(8):
        for v in range(-1, LT):
            for w in range(1, LT + 1):
                if v + w < U:
                    C[v + w] += F(r + 8 * v) @ G(8 * w - r)
        if full and r == 0:
            for w in range(1, LT):
                C[LT + w] += F(8 * LT) @ G(8 * w)
        if LT > 8 and r == 3:
            parts.append(C)
            C = C * 0
    return parts + [C]


@pytest.mark.parametrize("full,LT", [(True, x) for x in range(1, 11)] + [(False, x) for x in range(1, 17)])
def test_sums_are_exact(full, LT):
    parts = _counts(LT, full)
    N = 128 * LT
    total = sum(parts).reshape(-1)
    for c in range(len(total)):                 # every product of the column, once
        assert total[c] == min(c, N) - max(0, c - N) + 1
    for p in parts:                             # the carry digits' two products in a column are below 2^8 each
        p = p.reshape(-1).copy()
        p[N:] -= np.minimum(p[N:], 2)
        assert p.max() <= 1024

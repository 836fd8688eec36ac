"""FP32 factors whose 2x2 pivots give columns outside the FP32 range: the
a-posteriori threshold test has to see them as the FP64 arithmetic does."""
import numpy as np
import pytest

from spral_gb300 import ssids

pytestmark = pytest.mark.gpu


def _pairs(a, below):
    """64 x 64, one front: 16 pivots [[0, a], [a, 0]], then a unit diagonal;
    below: entries {(row, column): value} of the rows under the first block."""
    A = np.zeros((64, 64))
    for i in range(0, 32, 2):
        A[i + 1, i] = a
    A[range(32, 64), range(32, 64)] = 1.0
    for (i, j), x in below.items():
        A[i, j] = x
    n = 64
    ptr = np.concatenate([[0], np.cumsum(np.arange(n, 0, -1))]).astype(np.int64)
    row = np.concatenate([np.arange(j, n, dtype=np.int32) for j in range(n)])
    return ptr, row, np.concatenate([A[j:, j] for j in range(n)]), np.tril(A) + np.tril(A, -1).T


def _factor(p, r, v):
    ak = ssids.analyse(p, r, np.arange(64, dtype=np.int32))
    assert ak.nnodes == 1  # an APP block step of 32 columns comes first
    return ssids.factor(ak, v, ssids.Options(precision=ssids.PRECISION_MIXED))


@pytest.mark.parametrize("below", [{(40, 0): 1e20, (41, 1): 1e20}, {(40, 1): 1e20, (41, 0): 1e20},
                                   {(40, 0): 1e20, (40, 1): 1e20, (41, 0): 1e20}],
                         ids=["second", "first", "both"])
def test_gpu_fp32_overflowing_two_by_two_column_fails(below):
    """A multiplier of 1e39 in one column of a 2x2 pivot beside a zero in the
    other: the pivot is not accepted."""
    p, r, v, A = _pairs(1e-19, below)
    fk, inf = _factor(p, r, v)
    # 15 pairs [[0, a], [a, 0]] with one negative eigenvalue each; the other
    # two columns against rows 40 and 41, a saddle point, with two
    assert (inf.flag, inf.num_neg, inf.matrix_rank) == (0, 17, 64)
    L = fk.front(0)["L"]
    assert np.isfinite(L).all() and np.abs(np.tril(L, -1)).max() <= 100 * (1 + 1e-6)
    x = fk.solve(A @ np.ones(64))
    # the entries of A @ 1 round; FP32 factors otherwise
    assert np.abs(x - 1.0).max() <= 1e-5
    fk.free()

"""Fronts of small leaf subtrees at the ends of the FP64 range and beyond the
sizes that the default subtree rule gives them."""
import numpy as np
import pytest

from spral_gb300 import matrices as M, ssids
from test_gpu_tpp_search import _saddles

pytestmark = pytest.mark.gpu


# 2^0: the fast reciprocals; 2^505: outside their range; 2^525 and 2^-525: the
# determinant of a 2x2 pivot's inverse is a denormal number, or overflows
@pytest.mark.parametrize("e", [0, 505, 525, -525])
def test_gpu_two_by_two_pivots_at_the_ends_of_the_range(e):
    p, r, v = _saddles(3, 40, 15, 20, seed=1)
    n = len(p) - 1
    ak = ssids.analyse(p, r, np.arange(n, dtype=np.int32))
    b = M.sym_matvec(p, r, v, np.random.default_rng(2).standard_normal((n, 2)))
    fk, inf = ssids.factor(ak, np.ldexp(v, e), ssids.Options(small=1e-300))
    assert inf.num_two > 0
    x = fk.solve(b)
    # x 2^e solves the matrix with right-hand side b: the fixtures' bound
    assert M.scaled_bwd_error(p, r, v, np.ldexp(x, e), b).max() <= 5e-14
    fk.free()


def test_gpu_zero_threshold_of_either_sign():
    """small = -0.0 finds no entry below it, as small = 0.0."""
    k = 12
    p, r, v = M.laplacian_3d(k, shift=-0.3)
    ak = ssids.analyse(p, r, M.nd_order_grid(k, k, k))
    b = np.random.default_rng(1).standard_normal(k ** 3)
    xs = []
    for small in (0.0, -0.0):
        fk, inf = ssids.factor(ak, v, ssids.Options(small=small))
        assert (inf.flag, inf.matrix_rank) == (0, k ** 3)
        xs.append(fk.solve(b))
        fk.free()
    assert np.array_equal(xs[0], xs[1])


def _pairs(w, border, tiny):
    """Two blocks of w columns under a border, diagonally dominant: in a block,
    pairs of columns are coupled by `tiny` and by 0.5 in turn."""
    rng = np.random.default_rng(3)
    n = 2 * w + border
    ptr, row, val = [0], [], []
    for j in range(n):
        b, k = divmod(j, w)
        rows = np.arange(j, n) if j >= 2 * w else np.concatenate(
            [np.arange(j, (b + 1) * w), np.arange(2 * w, n)])
        vals = rng.uniform(-1, 1, len(rows))
        vals[0] = rng.uniform(1, 2) * (n if j >= 2 * w else 10)
        if j < 2 * w:
            vals[1:w - k] = 0.0
            if k % 2 == 0:
                vals[1] = tiny if k % 4 == 0 else 0.5
        row.append(rows.astype(np.int32))
        val.append(vals)
        ptr.append(ptr[-1] + len(rows))
    return np.array(ptr, np.int64), np.concatenate(row), np.concatenate(val)


@pytest.mark.parametrize("tiny", [0.0, 1e-12, 1e-30, 1e-90])
@pytest.mark.parametrize("nrhs", [1, 4])
def test_gpu_two_by_two_pivots_of_any_off_diagonal_entry(tiny, nrhs):
    """Pairs of columns coupled by a tiny entry, or by 0.5, and by nothing else: the pivot search
    takes them as 2x2 pivots (the 2x2 test comes first and asks nothing of that
    entry), whose contribution has to keep its digits whatever its size."""
    p, r, v = _pairs(40, 30, tiny)
    n = len(p) - 1
    ak = ssids.analyse(p, r, np.arange(n, dtype=np.int32))
    fk, inf = ssids.factor(ak, v)
    assert inf.flag == 0 and inf.num_two >= 40
    b = M.sym_matvec(p, r, v, np.random.default_rng(4).standard_normal((n, nrhs)))
    # a diagonally dominant matrix: rounding, n terms a sum
    assert M.scaled_bwd_error(p, r, v, fk.solve(b), b).max() <= n * 2.0 ** -52
    fk.free()


def test_gpu_balance_of_a_small_subtree_front_of_many_columns():
    """560 columns in a front that the caller's subtree rule makes a small one,
    pairs of the last ones scaled by 2^30 and 2^-30 in turn: its contribution
    keeps the border's entries."""

    class Wide(ssids.Options):
        def cpu_options(self):
            c = super().cpu_options()
            c.small_subtree_threshold = 10 ** 9
            return c

    w = 560
    p, r, v = _pairs(w, 30, 0.25)
    n = len(p) - 1
    s = np.ones(n)
    for b in range(2):
        s[b * w + 512:(b + 1) * w] = np.ldexp(1.0, np.where(np.arange(w - 512) % 4 < 2, 30, -30))
    b = M.sym_matvec(p, r, v, np.random.default_rng(5).standard_normal((n, 2)))
    ak = ssids.analyse(p, r, np.arange(n, dtype=np.int32))
    cols = np.repeat(np.arange(n), np.diff(p))
    # a threshold that takes the scaled columns (pairs by themselves) in any order
    fk, inf = ssids.factor(ak, v * s[r] * s[cols], Wide(u=1e-13))
    assert (inf.flag, inf.num_neg, inf.num_delay) == (0, 0, 0)
    x = s[:, None] * fk.solve(s[:, None] * b)
    # the unscaled matrix is diagonally dominant: rounding, n terms a sum
    assert M.scaled_bwd_error(p, r, v, x, b).max() <= n * 2.0 ** -52
    fk.free()

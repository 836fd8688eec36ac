"""The residual of a refined solve row by row: short and long rows in one
matrix, and a matrix's bits whatever is stacked beside it."""
import numpy as np
import pytest

from spral_gb300 import batch, matrices as M, ssids

pytestmark = pytest.mark.gpu


def _rows(n, long_rows, length, seed):
    """Diagonally dominant symmetric matrix: a tridiagonal band, and rows
    `long_rows` with about `length` further entries."""
    rng = np.random.default_rng(seed)
    ent = {}
    for j in range(n - 1):
        ent[j + 1, j] = rng.uniform(-1, 1)
    for i in long_rows:
        for j in rng.choice(n, min(length, n), replace=False):
            if i != j:
                ent[max(i, j), min(i, j)] = rng.uniform(-1, 1)
    deg = np.zeros(n)
    for (i, j), x in ent.items():
        deg[i] += abs(x)
        deg[j] += abs(x)
    for j in range(n):
        ent[j, j] = 1.01 * deg[j] * (1 if j % 3 else -1)
    keys = sorted(ent, key=lambda t: (t[1], t[0]))
    ptr = np.concatenate([[0], np.cumsum(np.bincount([j for _, j in keys], minlength=n))])
    return (ptr.astype(np.int64), np.array([i for i, _ in keys], np.int32),
            np.array([ent[k] for k in keys]))


def _mixed(nrhs):
    """Averages below and above 12 non-zeros a row, rows of 11 to 15, one dense row."""
    return [_rows(200, range(0, 200, 2), 30, 1), _rows(900, [], 0, 2), _rows(700, [3, 699], 700, 3),
            _rows(333, range(0, 333, 3), 11, 4), M.laplacian_2d(17, 19, -0.4)]


# one, and two chunks of right-hand sides
@pytest.mark.parametrize("nrhs", [1, 6])
def test_gpu_refined_bits_do_not_depend_on_the_batch(nrhs):
    mats = _mixed(nrhs)
    lens = [2 * len(v) - (len(p) - 1) for p, _, v in mats]
    sizes = [len(p) - 1 for p, _, _ in mats]
    assert lens[0] > 12 * sizes[0] and sum(lens) < 12 * sum(sizes)
    orders = [np.asarray(ssids.order_amd(p, r)) for p, r, _ in mats]
    opts = ssids.Options(precision=ssids.PRECISION_MIXED, max_refine=2, refine_tol=1e-300,
                         fp64_fallback=False)
    rng = np.random.default_rng(5)
    bs = [rng.standard_normal((n, nrhs)) for n in sizes]
    bak = batch.BatchAkeep([m[:2] for m in mats], orders)
    fk = ssids.Fkeep(bak.akeep, bak.stack_values([m[2] for m in mats]), opts)
    xs = bak.split(fk.solve_refined(bak.stack_rhs(bs)[0]))
    fk.free()
    for (p, r, v), order, b, x in zip(mats, orders, bs, xs):
        assert M.scaled_bwd_error(p, r, v, x, b).max() <= 1e-14
        alone = ssids.Fkeep(ssids.analyse(p, r, order), v, opts)
        assert np.array_equal(alone.solve_refined(b), x)
        alone.free()

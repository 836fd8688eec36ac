"""FP64 solves of three and more columns component by component: matrices and
solutions whose entries are far apart, and pivot blocks with large inverses.
One column at a time is solved by substitution in FP64 multiply-adds."""
import numpy as np
import pytest

from spral_gb300 import matrices as M, ssids

pytestmark = pytest.mark.gpu


def _grid(k, shift):
    p, r, v = M.laplacian_3d(k, shift=shift)
    return p, r, v, ssids.analyse(p, r, M.nd_order_grid(k, k, k))


def _cols(p):
    return np.repeat(np.arange(len(p) - 1), np.diff(p))


# separators of 484, 242, ... columns: several pivot blocks, contribution rows
@pytest.mark.parametrize("nrhs", [3, 9, 16])
def test_gpu_block_solve_follows_a_diagonal_scaling(nrhs):
    """Cholesky of S A S with S of powers of two from 2^-17 to 2^17: every
    operation scales exactly, so S x has the bits of the unscaled solution."""
    p, r, v, ak = _grid(22, 0.1)
    n = len(p) - 1
    rng = np.random.default_rng(nrhs)
    s = 2.0 ** rng.integers(-17, 18, n)
    b = rng.standard_normal((n, nrhs))
    f0, i0 = ssids.factor(ak, v, posdef=True)
    f1, i1 = ssids.factor(ak, v * s[r] * s[_cols(p)], posdef=True)
    assert i0.flag == 0 and i1.flag == 0
    for job in (0, 1, 3):
        x0 = f0.solve(b, job=job)
        # forward: L_chol^-1 (its D^(1/2) makes the result scale-free); backward
        # from there
        x1 = f1.solve(b if job == 3 else s[:, None] * b, job=job)
        assert np.array_equal(x1 if job == 1 else s[:, None] * x1, x0)
    f0.free()
    f1.free()


def test_gpu_block_solve_of_a_scaled_indefinite_matrix():
    p, r, v, ak = _grid(22, -0.3)
    n = len(p) - 1
    # from 1e-5 in one corner to 1e5 in the opposite one; neighbours differ by
    # 1.5 at most, so threshold pivoting finds its pivots as it does unscaled
    i = np.arange(n)
    s = 10.0 ** (10 * (i % 22 + i // 22 % 22 + i // 484) / 63.0 - 5)
    w = v * s[r] * s[_cols(p)]
    x0 = np.random.default_rng(2).standard_normal((n, 6))  # solution of the unscaled matrix
    b = M.sym_matvec(p, r, v, x0) * s[:, None]
    fk, inf = ssids.factor(ak, w)
    assert inf.flag == 0
    block = np.abs(s[:, None] * fk.solve(b) - x0).max(axis=0)
    alone = np.array([np.abs(s * fk.solve(b[:, q]) - x0[:, q]).max() for q in range(6)])
    # as the unscaled matrix' solves: rounding times a condition of about 1e3,
    # or the growth of threshold pivots that the columns alone have as well
    assert (block <= 1e-11 + 10 * alone).all()
    fk.free()


@pytest.mark.parametrize("nrhs", [4, 11])
def test_gpu_block_solve_of_decaying_solutions(nrhs):
    """Columns of the inverse of a diagonally dominant M-matrix decay to 1e-60
    and less; nothing cancels, so every component has a small relative error."""
    p, r, v, ak = _grid(22, 8.0)
    n = len(p) - 1
    fk, inf = ssids.factor(ak, v, posdef=True)
    assert inf.flag == 0
    b = np.zeros((n, nrhs))
    b[np.random.default_rng(3).choice(n, nrhs, replace=False), np.arange(nrhs)] = 1.0
    x = fk.solve(b)
    for q in range(nrhs):
        y = fk.solve(b[:, q])
        assert y.min() > 0 and y.min() < 1e-25
        # relative errors of 2^-47 a sum, some hundred sums on a path to the root
        # and back
        assert (np.abs(x[:, q] - y) <= 2000 * 2.0 ** -47 * y).all()
    fk.free()


def _dense_posdef(blk, n, seed):
    """L L^T with a unit lower L: `blk` below the diagonal in blocks of 32, small
    entries elsewhere; lower CSC with every entry stored."""
    rng = np.random.default_rng(seed)
    L = np.tril(0.02 * rng.standard_normal((n, n)), -1) + np.eye(n)
    for c in range(0, n, 32):
        e = min(c + 32, n)
        L[c:e, c:e] = np.tril(np.full((e - c, e - c), blk), -1) + np.eye(e - c)
    A = L @ L.T
    ptr = np.concatenate([[0], np.cumsum(np.arange(n, 0, -1))]).astype(np.int64)
    row = np.concatenate([np.arange(j, n, dtype=np.int32) for j in range(n)])
    return ptr, row, np.concatenate([A[j:, j] for j in range(n)])


# inverses of 1 to 3e4 in the blocks: below and above the bound for products
@pytest.mark.parametrize("blk", [-0.05, -0.25, -0.4])
def test_gpu_block_solve_with_growing_inverses(blk):
    p, r, v = _dense_posdef(blk, 230, seed=4)
    n = len(p) - 1
    ak = ssids.analyse(p, r, np.arange(n, dtype=np.int32))
    fk, inf = ssids.factor(ak, v, posdef=True)
    assert inf.flag == 0
    b = M.sym_matvec(p, r, v, np.random.default_rng(5).standard_normal((n, 5)))
    x = fk.solve(b)
    alone = np.stack([fk.solve(b[:, q]) for q in range(5)], axis=1)
    # the bound of the reference fixtures; substitution is backward stable
    # whatever the growth, and so are its blocks
    assert M.scaled_bwd_error(p, r, v, alone, b).max() <= 2e-15
    assert M.scaled_bwd_error(p, r, v, x, b).max() <= 2e-15
    fk.free()

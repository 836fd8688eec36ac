"""TPP fronts whose pivot search is carried out by every warp of a CTA: dense
saddle points whose first columns have no pivot among themselves, so that the
search runs through many candidates, and fronts of more than 1024 rows, whose
first candidate is examined by all warps too.  Every factorisation has to give
the same pivots, the oracle's in FP64."""
import numpy as np
import pytest

from spral_gb300 import matrices as M, ssids
import oracle

pytestmark = pytest.mark.gpu


def _saddles(nblk, w, n0, border, seed):
    """nblk dense saddle points [[0, B], [B^T, G]] of order w with every entry
    stored (a front each), n0 columns in the zero block, G diagonally dominant;
    all coupled to `border` last columns, also dominant.  Lower CSC."""
    rng = np.random.default_rng(seed)
    n = nblk * w + border
    ptr, row, val = [0], [], []
    for j in range(n):
        b, k = divmod(j, w)
        inner = np.arange(j, (b + 1) * w) if b < nblk else np.arange(j, n)
        rows = np.concatenate([inner, np.arange(nblk * w, n)]) if b < nblk else inner
        vals = rng.uniform(-1, 1, len(rows))
        if b < nblk and k < n0:
            vals[:n0 - k] = 0.0
        else:
            vals[0] = 2.0 * n + rng.uniform(0, 1)
        row.append(rows.astype(np.int32))
        val.append(vals)
        ptr.append(ptr[-1] + len(rows))
    return np.array(ptr, np.int64), np.concatenate(row), np.concatenate(val)


# small leaf subtrees (blocks under a border): 40 rows and more, of two and of
# eight warps, in shared memory; one front by itself: 300 rows, in place, and
# 1100, where all warps examine the first candidate too
@pytest.mark.parametrize("precision", [ssids.PRECISION_FP64, ssids.PRECISION_MIXED],
                         ids=["fp64", "mixed"])
@pytest.mark.parametrize("nblk,w,n0,border", [(3, 40, 15, 20), (3, 76, 35, 20), (3, 130, 60, 20),
                                              (1, 300, 140, 0), (1, 1100, 60, 0),
                                              (1, 1100, 300, 0)])
def test_gpu_tpp_search_by_all_warps_repeats(nblk, w, n0, border, precision):
    p, r, v = _saddles(nblk, w, n0, border, seed=w + n0)
    n = len(p) - 1
    ak = ssids.analyse(p, r, np.arange(n, dtype=np.int32))
    assert ak.nnodes == nblk  # the last block and the border are the root
    leaves = max(nblk - 1, 1)
    method = 2 if border else 3
    opts = ssids.Options(pivot_method=method, precision=precision)
    b = np.random.default_rng(n).standard_normal((n, 2))
    fk, inf = ssids.factor(ak, v, opts)
    # Sylvester's law: G is positive definite and B has full rank
    assert (inf.flag, inf.num_neg, inf.matrix_rank) == (0, nblk * n0, n)
    piv, d = fk.enquire_indef()
    x = fk.solve(b)
    perms = [fk.front(i)["perm"] for i in range(leaves)]
    for _ in range(6):
        assert fk.refactor(v) == 0
        q, e = fk.enquire_indef()
        assert np.array_equal(q, piv) and np.array_equal(e, d)
        assert np.array_equal(fk.solve(b), x)
    fk.free()
    # direct solves, FP64: the bound of the reference fixtures; FP32 factors:
    # FP32 rounding times the columns of a front
    bound = 5e-14 if precision == ssids.PRECISION_FP64 else 6e-8 * n
    assert M.scaled_bwd_error(p, r, v, x, b).max() <= bound
    if precision == ssids.PRECISION_FP64:
        F = oracle.OracleFactor(ak, v, options=oracle.default_options(pivot_method=method))
        for i in range(leaves):
            assert np.array_equal(perms[i], F.front(i)["perm"])

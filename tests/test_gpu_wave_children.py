"""The wavefront solves on a front with more children than a CTA has threads,
some of which hand it delayed columns: the wait for the children and the
search for a delayed column's child."""
import numpy as np
import pytest

from spral_gb300 import matrices as M, ssids

pytestmark = pytest.mark.gpu


def _arrow(nleaf, width, border, every, seed):
    """nleaf dense blocks of `width` columns, each coupled to `border` last
    columns; every `every`-th block ends in a column without a diagonal and
    without coupling inside the block, which no block can eliminate."""
    rng = np.random.default_rng(seed)
    n = nleaf * width + border
    ptr, row, val = [0], [], []
    for b in range(nleaf):
        for j in range(width):
            c = b * width + j
            alone = b % every == 0 and j == width - 1
            inner = [] if alone else [b * width + i for i in range(j, width)]
            if inner and b % every == 0:
                inner = [i for i in inner if i != b * width + width - 1]
            tail = list(range(nleaf * width, n))
            for i in inner + tail:
                row.append(i)
                if i == c:
                    val.append((width + border) * rng.choice([-1.0, 1.0]))
                else:
                    val.append(rng.uniform(-1, 1))
            ptr.append(len(row))
    for j in range(border):
        c = nleaf * width + j
        for i in range(c, n):
            row.append(i)
            val.append(nleaf * (1.0 if i == c else 0.01 * rng.uniform(-1, 1)))
        ptr.append(len(row))
    return (np.array(ptr, np.int64), np.array(row, np.int32), np.array(val))


@pytest.mark.parametrize("precision", [ssids.PRECISION_FP64, ssids.PRECISION_MIXED],
                         ids=["fp64", "mixed"])
@pytest.mark.parametrize("nleaf", [3, 257, 600])
def test_gpu_wave_many_children(nleaf, precision, monkeypatch):
    p, r, v = _arrow(nleaf, 34, 48, max(1, nleaf // 40), seed=nleaf)
    n = len(p) - 1
    ak = ssids.analyse(p, r, np.arange(n, dtype=np.int32))
    opts = ssids.Options(precision=precision)
    b = np.random.default_rng(3).standard_normal((n, 5))
    monkeypatch.setenv("SPRAL_GB300_SOLVE_WAVE", "1")
    fk, inf = ssids.factor(ak, v, opts)
    assert inf.flag == 0 and inf.num_delay > 0
    # direct solves: the fixtures' bound with FP64 factors, FP32 rounding times
    # the columns of a front and the pivot growth with FP32 factors
    bound = 5e-14 if precision == ssids.PRECISION_FP64 else 1e-3
    for q in (1, 5):
        x = fk.solve(b[:, :q])
        assert M.scaled_bwd_error(p, r, v, x, b[:, :q]).max() <= bound
    fk.free()
    monkeypatch.setenv("SPRAL_GB300_SOLVE_WAVE", "0")
    fs, _ = ssids.factor(ak, v, opts)
    y = fs.solve(b)
    assert M.scaled_bwd_error(p, r, v, y, b).max() <= bound
    fs.free()

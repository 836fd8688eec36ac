"""Refined solves with a NaN or Inf: the right-hand side (or the matrix of a
batch) that holds it has missed the target, the others are refined as without
it."""
import ctypes

import numpy as np
import pytest

from spral_gb300 import _native, batch, matrices as M, ssids

pytestmark = pytest.mark.gpu


def _refined(fk, b):
    torch = pytest.importorskip("torch")
    n, q = b.shape
    invp = fk.akeep.invp  # device arrays are in pivot order
    bd = torch.tensor(np.ascontiguousarray(b[invp].T), device="cuda")
    xd = torch.empty_like(bd)
    it, bwd = ctypes.c_int(0), ctypes.c_double(-1.0)
    assert _native.lib().spral_ssids_gpu_solve_refined_dev(
        fk.num, q, ctypes.c_void_p(bd.data_ptr()), ctypes.c_void_p(xd.data_ptr()), n,
        ctypes.byref(it), ctypes.byref(bwd)) == 0
    x = np.empty_like(b)
    x[invp] = xd.cpu().numpy().T
    return x, bwd.value


@pytest.mark.parametrize("precision", [ssids.PRECISION_FP64, ssids.PRECISION_MIXED],
                         ids=["fp64", "mixed"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_gpu_refined_solve_reports_non_finite_columns(precision, bad):
    p, r, v = M.laplacian_2d(30, 30, -0.5)
    ak = ssids.analyse(p, r, M.nd_order_grid(30, 30))
    fk, inf = ssids.factor(ak, v, ssids.Options(precision=precision, refine_tol=1e-14))
    assert inf.flag == 0
    b = np.random.default_rng(1).standard_normal((900, 3))
    x, bwd = _refined(fk, b)
    assert bwd <= 1e-14
    c = b.copy()
    c[17, 1] = bad
    y, bwd = _refined(fk, c)
    assert bwd == np.inf and not np.isfinite(y[:, 1]).all()
    assert M.scaled_bwd_error(p, r, v, y[:, [0, 2]], b[:, [0, 2]]).max() <= 1e-14
    assert fk.fallbacks == 0  # no factors make a solution of that column
    z = fk.solve_refined(c)
    assert np.isfinite(z[:, [0, 2]]).all() and not np.isfinite(z[:, 1]).all()
    fk.free()


def test_gpu_non_finite_solution_takes_the_fp64_fallback():
    """Entries above the FP32 range: the FP32 factors and the solution hold
    NaN, and the system is solved with FP64 factors."""
    n = 8
    A = np.diag(np.full(n, 2.0))
    A[n - 1, :2] = A[:2, n - 1] = 1e39
    ptr = np.concatenate([[0], np.cumsum(np.arange(n, 0, -1))]).astype(np.int64)
    row = np.concatenate([np.arange(j, n, dtype=np.int32) for j in range(n)])
    v = np.concatenate([A[j:, j] for j in range(n)])
    ak = ssids.analyse(ptr, row, np.arange(n, dtype=np.int32))
    fk, _ = ssids.factor(ak, v, ssids.Options(precision=ssids.PRECISION_MIXED, refine_tol=1e-12))
    b = A @ np.ones(n)
    x, bwd = _refined(fk, b[:, None])
    assert np.isfinite(x).all() and bwd <= 1e-12 and fk.fallbacks == 1
    fk.free()


def test_gpu_batch_with_a_non_finite_right_hand_side():
    rng = np.random.default_rng(2)
    sizes = [8, 12, 20, 9]
    mats = [M.laplacian_2d(k, k, -0.4) for k in sizes]
    bak = batch.BatchAkeep([m[:2] for m in mats], [M.nd_order_grid(k, k) for k in sizes])
    for precision in (ssids.PRECISION_FP64, ssids.PRECISION_MIXED):
        fk = batch.BatchFkeep(bak, [v for _, _, v in mats],
                              ssids.Options(precision=precision, refine_tol=1e-14))
        bs = [rng.standard_normal((k * k, 2)) for k in sizes]
        bs[2][5, 0] = np.nan
        ys = fk.solve_refined(bs)
        for i, (p, r, v) in enumerate(mats):
            q = slice(1, 2) if i == 2 else slice(0, 2)
            assert M.scaled_bwd_error(p, r, v, ys[i][:, q], bs[i][:, q]).max() <= 1e-14
        assert not np.isfinite(ys[2][:, 0]).all() and np.isfinite(ys[2][:, 1]).all()
        e = fk.group_errors()
        assert e[2] == np.inf and (e[[0, 1, 3]] <= 1e-14).all()
        fk.free()

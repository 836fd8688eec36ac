"""The FP64 trailing update from exact FP16 slice products
(spral_ssids_gpu_slice_gemm_f64) against extended-precision products, and the
FP64 factorisations that use it for contribution blocks and panels."""
import numpy as np
import pytest

from spral_gb300 import _native, matrices as M, ssids
import oracle

pytestmark = pytest.mark.gpu


def _update(A, B, C, reps=1):
    torch = pytest.importorskip("torch")
    (m, k), n = A.shape, B.shape[0]
    d = [torch.tensor(x.ravel(order="F"), device="cuda") for x in (A, B, C)]
    rc = _native.lib().spral_ssids_gpu_slice_gemm_f64(
        m, n, k, d[0].data_ptr(), m, d[1].data_ptr(), n, d[2].data_ptr(), m, reps, None)
    assert rc == 0
    return d[2].cpu().numpy().reshape(m, n, order="F")


def _check(A, B, C):
    got = _update(A, B, C)
    m, n = C.shape
    low = np.tril(np.ones((m, n), dtype=bool))
    assert np.array_equal(got[~low], C[~low])  # strictly upper part never written
    a, b = A.astype(np.longdouble), B.astype(np.longdouble)
    prod = a @ b.T
    ref = C - prod
    # two FP64 roundings (the product's and the difference's), the operands'
    # truncation at 2^-62 of the row scale (at most twice the row maximum) and
    # the 7 digit products of the first level left out, 2^-62 each; the
    # reference's own sums at 64 bits
    scale = np.abs(A).max(axis=1)[:, None] * np.abs(B).max(axis=1)[None, :]
    tol = 2.0 ** -52 * (np.abs(prod) + np.abs(ref)) + A.shape[1] * 9.2 * 2.0 ** -60 * scale
    tol += A.shape[1] * 2.0 ** -63 * (np.abs(a) @ np.abs(b).T)
    assert (np.abs(got - ref) <= tol)[low].all()


# tile edges (128 x 64), stage and chunk edges in k (32, 128), the split of
# the k range (2048), trapezoids with an odd number of tile columns
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (64, 64, 32), (65, 63, 31), (128, 128, 33),
                                   (129, 127, 127), (127, 127, 128), (257, 129, 129), (300, 1, 64),
                                   (200, 193, 40), (70, 65, 2081)])
def test_slice_gemm_matches_extended_precision(m, n, k):
    rng = np.random.default_rng(1000 * m + k)
    A, B = rng.standard_normal((m, k)), rng.standard_normal((n, k))
    _check(A, B, rng.standard_normal((m, n)))


def test_slice_gemm_row_scales_extremes_and_non_finite():
    rng = np.random.default_rng(3)
    m, n, k = 150, 140, 50
    # rows of very different sizes, a zero row, a denormal row, entries spread
    # over twenty orders of magnitude, digits at their bounds
    A = rng.standard_normal((m, k)) * 10.0 ** rng.uniform(-120, 120, (m, 1))
    B = rng.standard_normal((n, k)) * 10.0 ** rng.uniform(-120, 120, (n, 1))
    A[3] = 0.0
    A[7] = rng.integers(1, 1 << 20, k) * 5e-324
    A[9] *= 10.0 ** rng.uniform(-20, 0, k)
    A[11], B[11] = 1.0 - 2.0 ** -53, -(1.0 - 2.0 ** -53)
    C = rng.standard_normal((m, n))
    _check(A, B, C)
    # a non-finite operand row gives a non-finite row or column, the rest is untouched
    A[20, 5], B[30, 6] = np.inf, np.nan
    got = _update(A, B, C)
    low = np.tril(np.ones((m, n), dtype=bool))
    bad = np.zeros((m, n), dtype=bool)
    bad[20], bad[:, 30] = True, True
    assert np.isnan(got[bad & low]).all() and np.isfinite(got[~bad & low]).all()


def test_slice_gemm_is_deterministic_and_rejects_bad_arguments():
    rng = np.random.default_rng(5)
    A, B, C = (rng.standard_normal(s) for s in ((400, 90), (400, 90), (400, 400)))
    assert np.array_equal(_update(A, B, C, 3), _update(A, B, C, 3))
    f = _native.lib().spral_ssids_gpu_slice_gemm_f64
    assert f(4, 5, 1, None, 4, None, 5, None, 4, 1, None) == -1  # N > M
    assert f(4, 4, 1, None, 3, None, 4, None, 4, 1, None) == -1  # lda < M
    assert f(4, 4, 0, None, 4, None, 4, None, 4, 1, None) == 0


def _rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("kind", ["lap3d", "kkt", "posdef"])
def test_gpu_fp64_factors_match_simt_and_oracle(kind, monkeypatch):
    """FP64 factorisations (failed columns in the saddle point) against those
    with the SIMT contribution update and the oracle; a captured
    refactorisation repeats the bits."""
    if kind == "kkt":
        p, r, v = M.kkt(3000, 1500, seed=7)
        ak = ssids.analyse(p, r, ssids.order_amd(p, r))
        neg = 1500  # Sylvester: H SPD, A full row rank
    else:
        k = 24
        shift = -0.3 if kind == "lap3d" else 0.1
        p, r, v = M.laplacian_3d(k, shift=shift)
        ak = ssids.analyse(p, r, M.nd_order_grid(k, k, k))
        neg = M.laplacian_eig_count_3d(k, k, k, shift)[0]
    pos = kind == "posdef"
    b = np.random.default_rng(5).standard_normal((len(p) - 1, 3))
    fk, inf = ssids.factor(ak, v, posdef=pos)
    assert inf.flag == 0 and inf.num_neg == neg
    x = fk.solve(b)
    # direct solves: the bound of the reference fixtures
    assert M.scaled_bwd_error(p, r, v, x, b).max() <= 5e-14
    for _ in range(2):  # the second one replays the captured graph (no delays)
        assert fk.refactor(v) == 0
        assert np.array_equal(fk.solve(b), x)
    fk.free()
    monkeypatch.setenv("SPRAL_GB300_TENSOR_CORES", "0")
    f0, inf0 = ssids.factor(ak, v, posdef=pos)
    assert inf0.num_neg == neg
    x0 = f0.solve(b)
    f0.free()
    assert _rel(x, x0) < 1e-10
    if not pos:
        assert _rel(x, oracle.OracleFactor(ak, v, blas=True).solve(b)) < 1e-10
    if kind == "kkt":
        assert inf.num_two > 0 and inf.num_delay > 0


@pytest.mark.parametrize("nrhs", [3, 4, 8, 9, 16, 21])
@pytest.mark.parametrize("kind", ["lap3d", "kkt"])
def test_gpu_fp64_block_solves_match_columns(kind, nrhs):
    """Three and more right-hand sides at once (tensor-core products in the
    fronts that are not one small item) against one column at a time (FP64
    multiply-adds): columns 200 orders of magnitude apart, a zero column and
    one with a NaN that must stay in its column."""
    if kind == "kkt":
        p, r, v = M.kkt(3000, 1500, seed=7)
        ak = ssids.analyse(p, r, ssids.order_amd(p, r))
    else:
        k = 22  # separators of 484, 242, ... columns
        p, r, v = M.laplacian_3d(k, shift=-0.3)
        ak = ssids.analyse(p, r, M.nd_order_grid(k, k, k))
    n = len(p) - 1
    fk, inf = ssids.factor(ak, v, ssids.Options(precision=ssids.PRECISION_FP64))
    assert inf.flag == 0
    b = np.random.default_rng(9).standard_normal((n, nrhs))
    b[:, 0] *= 1e100
    b[:, 1] *= 1e-100
    b[:, 2] = 0.0
    for job in (0, 1, 3):
        x = fk.solve(b, job=job)
        assert np.array_equal(fk.solve(b, job=job), x)
        assert np.all(x[:, 2] == 0.0)
        for q in range(nrhs):
            if q != 2:
                # rounding differences times a condition number of about 1e3
                assert _rel(x[:, q], fk.solve(b[:, q], job=job)) < 1e-11
    x = fk.solve(b)
    # direct solves: the bound of the reference fixtures (0 / 0 for the zero column)
    nz = np.arange(nrhs) != 2
    assert M.scaled_bwd_error(p, r, v, x[:, nz], b[:, nz]).max() <= 5e-14
    bad = b.copy()
    bad[n // 2, nrhs - 1] = np.nan
    y = fk.solve(bad)
    assert np.isnan(y[:, nrhs - 1]).any()
    assert np.array_equal(y[:, :nrhs - 1], x[:, :nrhs - 1])
    fk.free()


@pytest.mark.parametrize("m,n", [(33, 33), (64, 40), (65, 64), (97, 65), (129, 96), (160, 33),
                                 (200, 128), (257, 160), (700, 600)])
def test_gpu_dense_front_reconstructs(m, n):
    """P A P^T = L D L^T + Schur complement on the lower part, entry by entry
    (fronts at the edges of the in-front update's 64 x 32 tiles and 32-column
    steps), through the allocating dense entry point."""
    torch = pytest.importorskip("torch")
    import ctypes
    from dense_cases import gen_sym_indef
    a = gen_sym_indef(m, np.random.default_rng(m + n))
    a_d = torch.tensor(np.asfortranarray(a).ravel(order="F"), device="cuda")
    d_d = torch.zeros(2 * n + 2, dtype=torch.float64, device="cuda")
    p_d = torch.arange(n, dtype=torch.int32, device="cuda")
    P = ctypes.c_void_p
    ne = _native.lib().spral_ssids_gpu_ldlt_app_factor(
        m, n, P(p_d.data_ptr()), P(a_d.data_ptr()), m, P(d_d.data_ptr()), 1.0,
        P(a_d.data_ptr() + 8 * (n * m + n)), m, ctypes.byref(oracle.default_options()), None)
    assert ne == n
    f = a_d.cpu().numpy().reshape(m, m, order="F")
    d = d_d.cpu().numpy()
    perm = np.concatenate([p_d.cpu().numpy(), np.arange(n, m)])
    L = np.tril(f, -1)[:, :n] + np.eye(m, n)
    S = np.zeros((m, m))
    S[n:, n:] = np.tril(f[n:, n:])
    D = np.zeros((n, n))
    i = 0
    while i < n:
        if i + 1 < n and np.isinf(d[2 * i + 2]):
            D[i:i + 2, i:i + 2] = np.linalg.inv([[d[2 * i], d[2 * i + 1]],
                                                 [d[2 * i + 1], d[2 * i + 3]]])
            i += 2
        else:
            D[i, i] = 1.0 / d[2 * i]
            i += 1
    low = np.tril(np.ones((m, m), dtype=bool))
    err = np.abs(L @ D @ L.T + S - a[np.ix_(perm, perm)])
    # the standard bound of an LDL^T factorisation, with the factors' own
    # magnitudes; 2x2 pivots invert D^{-1} with a condition of at most 1/0.01
    size = np.abs(L) @ np.abs(D) @ np.abs(L).T + np.abs(S)
    assert (err <= 8 * (n + 4) * 2.0 ** -53 * 100 * size)[low].all()
    assert np.median((err / size)[low]) <= 8 * (n + 4) * 2.0 ** -53

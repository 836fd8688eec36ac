"""Performance cases of the factorise-and-solve path: what a program that uses
this package asks of it, by entry point, size and precision.

Kinds of case
  front   one dense front through the C-ABI (ldlt_app_factor), device arrays;
  grid    a 2D or 3D Laplacian through one of three entry points:
            "dev"      a handle kept between calls: new values and right-hand
                       sides on the device (refactor_dev, solve_refined_dev);
            "host"     a handle kept between calls, host arrays (refactor, solve);
            "oneshot"  a new handle for every matrix, host arrays
                       (Fkeep, solve_refined, free);
  kkt     a saddle-point matrix (2x2 pivots, delayed columns), as "dev";
  batch   many small 2D Laplacians stacked into one forest (BatchFkeep).

Every sparse case solves A x = b with b = A x0 for a known x0.  The entries of
A and x0 are short binary fractions (multiples of 2^-12, or 2^-27 for the
regularisation of a saddle point), so b is exact in FP64 and x0 is the exact
solution.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from spral_gb300 import _native, batch, matrices as M, ssids

#: scaled backward error that refined solves are asked for
TARGET = 1e-14
Q = 4096.0  # entries are multiples of 1/Q


def listed():
    return [
        # one small front: a caller with its own tree; latency and launches
        dict(name="front_96", kind="front", m=96, n=40),
        # one large front, wide contribution block
        dict(name="front_2400", kind="front", m=2400, n=900),
        # the smallest sparse call: 64 x 64 grid, one right-hand side, host arrays
        dict(name="grid2d_64", kind="grid", mode="host", nx=64, ny=64, nz=1, nrhs=1,
             precision="fp64", posdef=False, coef="const"),
        # the headline problem: 48^3 grid, 8 right-hand sides, both precisions
        dict(name="grid3d_48", kind="grid", mode="dev", nx=48, ny=48, nz=48, nrhs=8,
             precision="fp64", posdef=False, coef="const"),
        dict(name="grid3d_48_mixed", kind="grid", mode="dev", nx=48, ny=48, nz=48, nrhs=8,
             precision="mixed", posdef=False, coef="const"),
        # the largest matrix of the serving mix, many right-hand sides
        dict(name="grid3d_57", kind="grid", mode="dev", nx=57, ny=57, nz=57, nrhs=40,
             precision="fp64", posdef=False, coef="var"),
        # a matrix factored once (the plain analyse/factor/solve sequence), ragged grid
        dict(name="oneshot_23", kind="grid", mode="oneshot", nx=23, ny=19, nz=26, nrhs=3,
             precision="fp64", posdef=False, coef="var"),
        # Cholesky of an implicit time step: values change, pattern stays
        dict(name="posdef_33", kind="grid", mode="host", nx=33, ny=33, nz=31, nrhs=2,
             precision="fp64", posdef=True, coef="var"),
        # saddle points: an interior-point iteration's system, both precisions
        dict(name="kkt_6000", kind="kkt", nh=4000, na=2000, nrhs=4, precision="fp64"),
        dict(name="kkt_15000_mixed", kind="kkt", nh=10000, na=5000, nrhs=8, precision="mixed"),
        # many small independent matrices, both precisions
        dict(name="batch_320", kind="batch", count=320, lo=8, hi=128, precision="fp64"),
        dict(name="batch_320_mixed", kind="batch", count=320, lo=8, hi=128, precision="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["front", "grid2d", "grid3d", "grid3d", "kkt", "batch"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "front":
        m = _log(rng, 24, 2400)
        return dict(kind="front", m=m, n=_log(rng, min(16, m), min(m, 1000)))
    if kind == "kkt":
        nh = _log(rng, 300, 10000 if precision == "mixed" else 5000)
        return dict(kind="kkt", nh=nh, na=nh // 2, nrhs=rng.randint(1, 8), precision=precision)
    if kind == "batch":
        return dict(kind="batch", count=_log(rng, 24, 320), lo=8, hi=_log(rng, 24, 128),
                    precision=precision)
    mode = rng.choice(["dev", "host", "oneshot"])
    # unrefined solves and Cholesky are for FP64 factors
    if mode == "host":
        precision = "fp64"
    case = dict(kind="grid", mode=mode, precision=precision,
                posdef=mode == "host" and rng.random() < 0.5,
                coef=rng.choice(["const", "var"]), nrhs=_log(rng, 1, 40))
    if kind == "grid2d":
        return dict(case, nx=_log(rng, 16, 300), ny=_log(rng, 16, 300), nz=1)
    side = _log(rng, 10, 54)
    return dict(case, nx=side, ny=max(8, side - rng.randint(0, 5)),
                nz=max(8, side - rng.randint(-3, 5)))


# ---------------------------------------------------------------- matrices
def _ints(rng, lo, hi, size):
    """Uniform multiples of 1/Q in [lo, hi]."""
    return rng.integers(int(lo * Q), int(hi * Q) + 1, size) / Q


def _normals(rng, size):
    return np.round(rng.standard_normal(size) * Q) / Q


@functools.lru_cache(maxsize=32)
def _grid_plan(nx, ny, nz):
    """Pattern and analyse of a grid: kept by a program for all its values."""
    if nz == 1:
        ptr, row, _ = M.laplacian_2d(nx, ny)
    else:
        ptr, row, _ = M.laplacian_3d(nx, ny, nz)
    return ptr, row, ssids.analyse(ptr, row, M.nd_order_grid(nx, ny, nz))


@functools.lru_cache(maxsize=8)
def _kkt_plan(nh, na):
    ptr, row, _ = M.kkt(nh, na, seed=2026)
    return ptr, row, ssids.analyse(ptr, row, ssids.order_amd(ptr, row))


@functools.lru_cache(maxsize=8)
def _batch_plan(count, lo, hi):
    rng = np.random.default_rng(4096)
    sides = np.exp(rng.uniform(np.log(lo), np.log(hi + 1), count)).astype(int)
    pats, orders = {}, {}
    for k in set(sides.tolist()):
        pats[k] = M.laplacian_2d(k, k)[:2]
        orders[k] = M.nd_order_grid(k, k)
    bak = batch.BatchAkeep([pats[k] for k in sides], [orders[k] for k in sides])
    return sides, bak


def _cols(ptr):
    return np.repeat(np.arange(len(ptr) - 1), np.diff(ptr))


def _grid_values(case, seed):
    """Indefinite: shift in [-0.5, 0] (3D) or [-1, 0] (2D) of the Laplacian;
    "var": edge weights in [0.75, 1.25] instead of 1.  Positive definite: a
    positive shift, as an implicit time step has."""
    ptr, row, _ = _grid_plan(case["nx"], case["ny"], case["nz"])
    rng = np.random.default_rng([seed, 1])
    n, cols = len(ptr) - 1, _cols(ptr)
    off = row != cols
    if case["posdef"]:
        shift = _ints(rng, 0.01, 0.5, 1)[0]
    else:
        shift = -_ints(rng, 0.05, 1.0 if case["nz"] == 1 else 0.5, 1)[0]
    degree = 4.0 if case["nz"] == 1 else 6.0
    val = np.where(off, -1.0, degree + shift)
    if case["coef"] == "var":
        w = _ints(rng, 0.75, 1.25, int(off.sum()))
        val[off] = -w
        # Dirichlet boundary edges keep weight 1
        d = np.bincount(cols[off], w - 1.0, n) + np.bincount(row[off], w - 1.0, n)
        val[~off] += d[cols[~off]]
    return val


def _kkt_values(case, seed):
    """[[H, A^T], [A, -2^-27 I]]: N(0, 1) entries, H diagonally dominant."""
    nh = case["nh"]
    ptr, row, _ = _kkt_plan(nh, case["na"])
    rng = np.random.default_rng([seed, 1])
    n, cols = len(ptr) - 1, _cols(ptr)
    off = row != cols
    val = _normals(rng, len(row))
    inh = off & (row < nh)
    s = np.bincount(cols[inh], np.abs(val[inh]), n) + np.bincount(row[inh], np.abs(val[inh]), n)
    val[~off] = np.where(cols[~off] < nh, s[cols[~off]] + 1.0, -(2.0 ** -27))
    return val


def _batch_values(case, seed):
    """Shifts in [-1, 0], none closer than 1e-4 to an eigenvalue."""
    sides, bak = _batch_plan(case["count"], case["lo"], case["hi"])
    rng = np.random.default_rng([seed, 1])
    vals = []
    for k, (ptr, row) in zip(sides.tolist(), bak.patterns):
        shift = -_ints(rng, 0.0, 1.0, 1)[0]
        while M.laplacian_eig_count_2d(k, k, shift)[2] < 1e-4:
            shift = -_ints(rng, 0.0, 1.0, 1)[0]
        vals.append(np.where(row == _cols(ptr), 4.0 + shift, -1.0))
    return vals


def _solution(n, nrhs, seed):
    return _normals(np.random.default_rng([seed, 2]), (n, nrhs))


def _times(ptr, row, val, x):
    """A x on the GPU (every sum is exact), n x nrhs, as a device array."""
    dev = torch.device("cuda")
    r = torch.as_tensor(np.asarray(row, dtype=np.int64), device=dev)
    c = torch.as_tensor(_cols(ptr), device=dev)
    v = torch.as_tensor(val, device=dev)[:, None]
    xd = torch.as_tensor(x, device=dev)
    y = torch.zeros_like(xd)
    y.index_add_(0, r, v * xd[c])
    off = r != c
    y.index_add_(0, c[off], v[off] * xd[r[off]])
    return y


# ---------------------------------------------------------------- fronts
def _front_matrix(case, seed):
    """Random symmetric, Unif[-1, 1], as a dense front of a general matrix."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    m = case["m"]
    a = torch.rand((m, m), generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    return torch.tril(a) + torch.tril(a, -1).T


class _Front:
    def __init__(self, case, seed):
        self.m, self.n = case["m"], case["n"]
        m, n = self.m, self.n
        a = _front_matrix(case, seed)
        # column-major: row k of the tensor is column k of the front
        self.a0 = a[:n].contiguous()
        self.s0 = a[n:, n:].contiguous()
        self.perm0 = torch.arange(n, dtype=torch.int32, device="cuda")
        self.a, self.s = torch.empty_like(self.a0), torch.empty_like(self.s0)
        self.perm = torch.empty_like(self.perm0)
        self.d = torch.zeros(2 * n + 2, dtype=torch.float64, device="cuda")
        self.stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        self.lib = _native.lib()

    def run(self):
        m, n = self.m, self.n
        self.a.copy_(self.a0)
        self.s.copy_(self.s0)
        self.perm.copy_(self.perm0)
        p = ctypes.c_void_p
        ne = self.lib.spral_ssids_gpu_ldlt_app_factor(
            m, n, p(self.perm.data_ptr()), p(self.a.data_ptr()), m, p(self.d.data_ptr()), 1.0,
            p(self.s.data_ptr()) if m > n else None, max(m - n, 1), None, self.stream)
        # D is finite but for the marks of 2x2 pivots; L is the lower part
        out = {"nelim": ne, "perm": self.perm, "d": self.d[:2 * n], "l": self.a}
        if m > n:
            out["schur"] = self.s
        return out


# ---------------------------------------------------------------- sparse
def _options(case):
    return ssids.Options(precision=ssids.PRECISION_MIXED if case["precision"] == "mixed"
                         else ssids.PRECISION_FP64, max_refine=20, refine_tol=TARGET)


class _Dev:
    """A handle kept on the device; values and right-hand sides arrive there."""

    def __init__(self, case, ptr, row, ak, values, seed):
        val = values(case, seed)
        self.ak, self.nrhs = ak, case["nrhs"]
        # the handle was made for the values of an earlier step
        self.fk = ssids.Fkeep(ak, values(case, seed + 7919), _options(case))
        b = _times(ptr, row, val, _solution(ak.n, self.nrhs, seed))
        invp = torch.as_tensor(ak.invp.astype(np.int64), device="cuda")
        self.val = torch.as_tensor(val, device="cuda")
        self.b = b[invp].T.contiguous()  # pivot order, one row per right-hand side
        self.x = torch.empty_like(self.b)
        self.it, self.bwd = ctypes.c_int(0), ctypes.c_double(0)
        self.lib = _native.lib()
        torch.cuda.synchronize()

    def run(self):
        flag = self.fk.refactor_dev(self.val.data_ptr())
        p = ctypes.c_void_p
        rc = self.lib.spral_ssids_gpu_solve_refined_dev(
            self.fk.num, self.nrhs, p(self.b.data_ptr()), p(self.x.data_ptr()), self.ak.n,
            ctypes.byref(self.it), ctypes.byref(self.bwd))
        inf = self.fk.inform
        return {"x": self.x, "status": [flag, rc, inf.num_neg, inf.matrix_rank]}


class _Host:
    """A handle kept on the device, host arrays in and out."""

    def __init__(self, case, ptr, row, ak, values, seed):
        self.val = values(case, seed)
        self.fk = ssids.Fkeep(ak, values(case, seed + 7919), _options(case),
                              posdef=case["posdef"])
        self.b = _times(ptr, row, self.val, _solution(ak.n, case["nrhs"], seed)).cpu().numpy()

    def run(self):
        flag = self.fk.refactor(self.val)
        x = self.fk.solve(self.b)
        inf = self.fk.inform
        return {"x": x, "status": [flag, inf.num_neg, inf.matrix_rank]}


class _OneShot:
    """analyse is kept; every matrix gets a handle of its own."""

    def __init__(self, case, ptr, row, ak, values, seed):
        self.ak, self.opts = ak, _options(case)
        self.val = values(case, seed)
        self.b = _times(ptr, row, self.val, _solution(ak.n, case["nrhs"], seed)).cpu().numpy()

    def run(self):
        fk = ssids.Fkeep(self.ak, self.val, self.opts)
        x = fk.solve_refined(self.b)
        inf = fk.inform
        fk.free()
        return {"x": x, "status": [inf.flag, inf.num_neg, inf.matrix_rank]}


class _Batch:
    def __init__(self, case, seed):
        _, self.bak = _batch_plan(case["count"], case["lo"], case["hi"])
        self.vals = _batch_values(case, seed)
        self.fk = batch.BatchFkeep(self.bak, _batch_values(case, seed + 7919), _options(case))
        val = self.bak.stack_values(self.vals)
        b = _times(self.bak.ptr, self.bak.row, val, _solution(self.bak.n, 1, seed))
        invp = torch.as_tensor(self.bak.akeep.invp.astype(np.int64), device="cuda")
        self.b = b[invp, 0].contiguous()
        self.x = torch.empty_like(self.b)
        torch.cuda.synchronize()

    def run(self):
        flag = self.fk.refactor(self.vals)
        self.fk.solve_refined_dev(self.b, self.x)
        inertia = self.fk.inertia()
        # negative and zero pivots of every matrix (2x2 counts depend on ties)
        return {"x": self.x, "flag": flag, "inertia": np.ascontiguousarray(inertia[:, [0, 2]])}


def prepare(case, seed):
    if case["kind"] == "front":
        return _Front(case, seed)
    if case["kind"] == "batch":
        return _Batch(case, seed)
    if case["kind"] == "kkt":
        return _Dev(case, *_kkt_plan(case["nh"], case["na"]), _kkt_values, seed)
    make = {"dev": _Dev, "host": _Host, "oneshot": _OneShot}[case["mode"]]
    return make(case, *_grid_plan(case["nx"], case["ny"], case["nz"]), _grid_values, seed)


def run(state):
    return state.run()


# ---------------------------------------------------------------- accounting
def _akeep(case):
    if case["kind"] == "batch":
        return _batch_plan(case["count"], case["lo"], case["hi"])[1].akeep
    if case["kind"] == "kkt":
        return _kkt_plan(case["nh"], case["na"])[2]
    return _grid_plan(case["nx"], case["ny"], case["nz"])[2]


def work(case):
    """Factorisation: the square of every column's count, a multiplication and
    an addition to each pair of entries of the lower triangle.  Solve: two
    passes over the factors.  Bytes: values and right-hand sides in, the
    solution out (fronts: the lower part in, L, D and the update out)."""
    if case["kind"] == "front":
        m, n = case["m"], case["n"]
        low = n * (n + 1) // 2 + (m - n) * n + (m - n) * (m - n + 1) // 2
        return {"bytes": 2 * 8 * low + 16 * n + 8 * n,
                "flops": float(sum((m - k) ** 2 for k in range(n)))}
    ak = _akeep(case)
    nrow, ncol = ak.front_sizes()
    flops = fact = 0.0
    for k in range(int(ncol.max())):
        live = (nrow - k)[ncol > k].astype(np.float64)
        flops += float((live * live).sum())
        fact += float(live.sum())
    nrhs = case.get("nrhs", 1)
    return {"bytes": 8 * (ak.nnz + 2 * ak.n * nrhs), "flops": flops + 4.0 * fact * nrhs}


def exact(case, seed):
    if case["kind"] == "front":
        m, n = case["m"], case["n"]
        out = {"nelim": None, "perm": None, "d": None, "l": None}
        if m > n:
            # the Schur complement does not depend on the pivots; the entry
            # point updates its lower triangle (upper in row-major terms)
            a = _front_matrix(case, seed)
            s = a[n:, n:] - a[n:, :n] @ torch.linalg.solve(a[:n, :n], a[:n, n:])
            out["schur"] = torch.triu(s) + torch.tril(a[n:, n:], -1)
        return out
    ak = _akeep(case)
    if case["kind"] == "batch":
        x0 = _solution(ak.n, 1, seed)
        return {"x": x0[ak.invp, 0], "flag": None, "inertia": None}
    x0 = _solution(ak.n, case["nrhs"], seed)
    if case["kind"] == "kkt" or case["mode"] == "dev":
        x0 = np.ascontiguousarray(x0[ak.invp].T)
        return {"x": x0, "status": [None] * 4}
    return {"x": x0, "status": [None] * 3}

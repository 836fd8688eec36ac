"""Allocations that fail at every point of a factorisation and of a solve (the
n-th allocation of the library fails once): the call reports it or does
without, and the handle works afterwards."""
import numpy as np
import pytest

from spral_gb300 import _native, matrices as M, ssids

pytestmark = pytest.mark.gpu


def _problem():
    p, r, v = M.laplacian_3d(14, shift=-0.3)
    ak = ssids.analyse(p, r, M.nd_order_grid(14, 14, 14))
    b = np.random.default_rng(1).standard_normal((len(p) - 1, 4))
    return p, r, v, ak, b


@pytest.fixture
def fail_after():
    lib = _native.lib()
    yield lib.spral_ssids_gpu_inject_alloc_failure
    lib.spral_ssids_gpu_inject_alloc_failure(-1)


def _check(fk, p, r, v, b):
    # direct solve, FP64: the bound of the reference fixtures; FP32 factors: the
    # same bound in units of their precision
    tol = 5e-14 * (2.0 ** 29 if fk.options.precision == ssids.PRECISION_MIXED else 1.0)
    assert M.scaled_bwd_error(p, r, v, fk.solve(b), b).max() <= tol


@pytest.mark.parametrize("precision", [ssids.PRECISION_FP64, ssids.PRECISION_MIXED],
                         ids=["fp64", "mixed"])
def test_gpu_handle_works_after_a_failed_allocation(fail_after, precision):
    p, r, v, ak, b = _problem()
    opts = ssids.Options(precision=precision)
    ssids.factor(ak, v, opts)[0].free()  # the device's one-time measurements
    reported = 0
    for k in range(40):
        fail_after(k)
        try:
            fk, inf = ssids.factor(ak, v, opts)
        except RuntimeError:
            continue  # no handle
        finally:
            fail_after(-1)
        if inf.flag != 0:
            assert inf.flag == ssids.SSIDS_ERROR_ALLOCATION
            reported += 1
            assert fk.refactor(v) == 0
        _check(fk, p, r, v, b)
        fk.free()
    assert reported > 0
    fk, inf = ssids.factor(ak, v, opts)
    assert inf.flag == 0
    for k in range(20):
        # values anew, so that the solve prepares its tables anew
        assert fk.refactor(v) == 0
        fail_after(k)
        try:
            fk.solve(b)
        except RuntimeError:
            pass
        fail_after(-1)
        _check(fk, p, r, v, b)
    fk.free()


def test_gpu_slices_are_given_up_for_memory_the_factorisation_needs(fail_after):
    """FP64 factors: from the first digit slices of the tensor-core updates on,
    an allocation that fails costs those and not the factorisation, and later
    factorisations and solves (captured graphs too) go on without."""
    p, r, v, ak, b = _problem()
    lib = _native.lib()
    flags = []
    for k in range(40):
        lib.spral_ssids_gpu_release_cache()
        fail_after(k)
        try:
            fk, inf = ssids.factor(ak, v)
        except RuntimeError:
            flags.append(None)
            continue
        finally:
            fail_after(-1)
        flags.append(inf.flag)
        if inf.flag == 0:
            _check(fk, p, r, v, b)
            for _ in range(2):
                assert fk.refactor(v) == 0
                _check(fk, p, r, v, b)
        fk.free()
    assert flags.count(ssids.SSIDS_ERROR_ALLOCATION) > 0 and flags[-1] == 0
    assert all(f == 0 for f in flags[flags.index(0):])


def test_gpu_solve_gives_up_slices_for_its_own_memory(fail_after):
    p, r, v, ak, b = _problem()
    lib = _native.lib()
    for refined in (False, True):
        for k in range(12):
            fk, inf = ssids.factor(ak, v)
            assert inf.flag == 0
            lib.spral_ssids_gpu_release_cache()
            fail_after(k)
            x = fk.solve_refined(b) if refined else fk.solve(b)
            fail_after(-1)
            assert M.scaled_bwd_error(p, r, v, x, b).max() <= 5e-14
            assert fk.refactor(v) == 0
            _check(fk, p, r, v, b)
            fk.free()

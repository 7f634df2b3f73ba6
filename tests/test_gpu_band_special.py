"""Band systems that hold NaN or infinities, through strut_gpu_band_solve_noalloc, in every variant of the
factorisation (one row set a warp, four warps, eight, and the rows without room for the zeros behind
the band).  BandGeneral's pivot search compares magnitudes strictly (linear_solver_backend.mojo:
640-657), so a NaN is never a candidate and never gives way: the elimination goes on and the status is
0, with a solution that is NaN wherever IEEE arithmetic makes it one."""
import numpy as np
import pytest

from strut_b200 import _abi as A
from tests.test_gpu_band_solve import _solve, _system

pytestmark = pytest.mark.gpu

SIZES = [(40, 1), (40, 12), (60, 20), (60, 24), (70, 31), (90, 40), (130, 62), (130, 63)]


def _band(K, bw):
    n = K.shape[0]
    band = np.zeros((n, 2 * bw + 1))
    for i in range(n):
        j = np.arange(max(0, i - bw), min(n, i + bw + 1))
        band[i, j - i + bw] = K[i, j]
    return band


@pytest.mark.parametrize("n,bw", SIZES)
@pytest.mark.parametrize("below", [0, 1])  # the diagonal; the entry under it
def test_nan_entry(n, bw, below):
    K, rhs = _system(n, bw, n + bw)
    c = n // 2
    K[c + below, c] = np.nan
    x, st = _solve(_band(K, bw), n, bw, A.SYSTEM_BAND_GENERAL, rhs)
    assert st == A.STRUT_OK
    assert np.isnan(x).all()  # every unknown depends on the one that is NaN


def _ieee_solve(K, bw, rhs, spd):
    """The reference's elimination (no interchange needed) and substitutions with IEEE divisions: a zero
    multiplier skips its row (linear_solver_backend.mojo:658-680, 735-812)."""
    n = K.shape[0]
    M, w = K.copy(), rhs.copy()
    with np.errstate(all="ignore"):
        for k in range(n):
            end = min(n, k + bw + 1)
            if spd:
                assert M[k, k] > 0.0
                M[k, k] = np.sqrt(M[k, k])
                M[k + 1:end, k] /= M[k, k]
                for i in range(k + 1, end):
                    M[i, k + 1:i + 1] -= M[i, k] * M[k + 1:i + 1, k]
                w[k] /= M[k, k]
            else:
                assert not np.any(np.abs(M[k + 1:end, k]) > abs(M[k, k])) and not abs(M[k, k]) <= 1e-14
                M[k + 1:end, k] /= M[k, k]
                for i in range(k + 1, end):
                    if M[i, k] != 0.0:
                        M[i, k + 1:end] -= M[i, k] * M[k, k + 1:end]
            w[k + 1:end] -= M[k + 1:end, k] * w[k]
        x = w.copy()
        for i in range(n - 1, -1, -1):
            if spd:
                x[i] /= M[i, i]
                j = max(0, i - bw)
                x[j:i] -= M[i, j:i] * x[i]
            else:
                for j in range(i + 1, min(n, i + bw + 1)):
                    x[i] -= M[i, j] * x[j]
                x[i] /= M[i, i]
    return x


def _special(kind, n, bw):
    K, rhs = _system(n, bw, 3 * n + bw)
    c = n // 2
    if kind == "inf_pivot":
        K[c, c] = np.inf
    elif kind == "huge_pivot":  # its reciprocal is subnormal
        K[c, c] = 1.5e308
    elif kind == "inf_rhs":
        rhs[c] = -np.inf
    elif kind == "overflow":  # unknowns beyond the largest number around c
        K *= 1e-10
        rhs[c] = 1e300
    else:  # a row that no row below it takes up
        K[c + 1:, c] = 0.0
        K[c, c + 1] = {"nan_upper": np.nan, "inf_upper": np.inf}[kind]
    return K, rhs


@pytest.mark.parametrize("n,bw", SIZES)
@pytest.mark.parametrize("kind,spd", [("inf_pivot", False), ("huge_pivot", False), ("inf_rhs", False),
                                      ("overflow", False), ("nan_upper", False), ("inf_upper", False),
                                      ("inf_pivot", True), ("huge_pivot", True), ("inf_rhs", True),
                                      ("overflow", True)])
def test_infinities(n, bw, kind, spd):
    """NaN and infinities where IEEE divisions put them; the finite unknowns to 1e-12 of the largest
    (as in test_band_solve, times ten for the mixed scales)."""
    K, rhs = _special(kind, n, bw)
    want = _ieee_solve(K, bw, rhs, spd)
    band = _band(K, bw)
    if spd:
        band = np.ascontiguousarray(band[:, bw::-1])
    x, st = _solve(band, n, bw, A.SYSTEM_BAND_SPD if spd else A.SYSTEM_BAND_GENERAL, rhs)
    assert st == A.STRUT_OK
    assert np.array_equal(np.isnan(x), np.isnan(want))
    assert np.array_equal(np.where(np.isinf(x), x, 0.0), np.where(np.isinf(want), want, 0.0))
    ok = np.isfinite(want)
    if ok.any():
        assert np.max(np.abs(x[ok] - want[ok])) <= 1e-12 * np.max(np.abs(want[ok]))


@pytest.mark.parametrize("n,bw", SIZES)
def test_slots_outside_the_matrix_do_not_count(n, bw):
    K, rhs = _system(n, bw, n - bw)
    band = _band(K, bw)
    x, st = _solve(band, n, bw, A.SYSTEM_BAND_GENERAL, rhs)
    for i in range(n):
        j = i + np.arange(-bw, bw + 1)
        band[i, (j < 0) | (j >= n)] = np.nan
    x2, st2 = _solve(band, n, bw, A.SYSTEM_BAND_GENERAL, rhs)
    assert st == st2 == A.STRUT_OK and np.array_equal(x, x2)

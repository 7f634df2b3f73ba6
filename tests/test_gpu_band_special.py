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

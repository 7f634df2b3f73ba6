"""The band factor-solve in shared memory at the edges of its variants (half bands 12, 16, 20, 31,
62, and bands that leave no room for the rows of zeros behind them),
through strut_gpu_band_solve_noalloc, against a dense solve in numpy.

The systems are diagonally dominant (condition number below 10), so a backward-stable elimination
is within a small multiple of n eps of the exact solution: 1e-13 of the largest entry for n <= 512.
"""
import ctypes as C

import numpy as np
import pytest

from strut_b200 import _abi as A

pytestmark = pytest.mark.gpu


def _system(n, bw, seed):
    rng = np.random.default_rng(seed)
    K = rng.standard_normal((n, n))
    K = K + K.T
    i = np.arange(n)
    K[np.abs(i[:, None] - i[None, :]) > bw] = 0.0
    K += np.diag(1.5 * np.abs(K).sum(1) + 1.0)
    return K, rng.standard_normal(n)


def _solve(band, n, bw, system, rhs):
    import torch
    from strut_b200 import runtime

    b, r = torch.from_numpy(band).cuda(), torch.from_numpy(rhs).cuda()
    x = torch.full((n,), np.nan, dtype=torch.float64, device="cuda")
    st = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    rc = runtime.lib().strut_gpu_band_solve_noalloc(C.c_void_p(b.data_ptr()), n, bw, system,
                                                    C.c_void_p(r.data_ptr()), C.c_void_p(x.data_ptr()),
                                                    C.c_void_p(st.data_ptr()),
                                                    C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == A.STRUT_OK
    return x.cpu().numpy(), int(st.item())


@pytest.mark.parametrize("n,bw", [(1, 0), (2, 1), (7, 3), (8, 7), (9, 8), (31, 11), (32, 12), (33, 13), (40, 16),
                                  (65, 17), (216, 20), (100, 21), (64, 24), (257, 24), (500, 24), (64, 25),
                                  (50, 31), (50, 32), (512, 25), (500, 25),
                                  (120, 40), (100, 61), (100, 62), (100, 63)])
@pytest.mark.parametrize("spd", [False, True])
def test_band_solve(n, bw, spd):
    K, rhs = _system(n, bw, 100 * n + bw)
    band = np.zeros((n, bw + 1 if spd else 2 * bw + 1))
    for i in range(n):
        for j in range(max(0, i - bw), min(n, i + bw + 1)):
            if not spd:
                band[i, j - i + bw] = K[i, j]
            elif j <= i:
                band[i, i - j] = K[i, j]
    ref = np.linalg.solve(K, rhs)
    x, st = _solve(band, n, bw, A.SYSTEM_BAND_SPD if spd else A.SYSTEM_BAND_GENERAL, rhs)
    assert st == 0
    assert np.abs(x - ref).max() <= 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("n,bw,col", [(40, 12, 0), (40, 12, 39 - 1), (90, 20, 33), (90, 24, 40), (90, 30, 40),
                                      (90, 30, 75)])
def test_band_solve_row_swap(n, bw, col):
    """A sub-diagonal entry larger than its pivot at `col` sends BandGeneral to partial pivoting."""
    K, rhs = _system(n, bw, n + col)
    K[col + 1, col] = 40.0 * np.abs(K).max()
    band = np.zeros((n, 2 * bw + 1))
    for i in range(n):
        for j in range(max(0, i - bw), min(n, i + bw + 1)):
            band[i, j - i + bw] = K[i, j]
    ref = np.linalg.solve(K, rhs)
    x, st = _solve(band, n, bw, A.SYSTEM_BAND_GENERAL, rhs)
    assert st == 0
    assert np.abs(x - ref).max() <= 1e-10 * np.abs(ref).max()


@pytest.mark.parametrize("col", [0, 7, 8, 39])
def test_band_solve_singular(col):
    """A zero column with nothing below it to swap in is singular at its own step."""
    n, bw = 40, 12
    K, rhs = _system(n, bw, col)
    K[:, col] = 0.0
    K[col, :] = 0.0
    band = np.zeros((n, 2 * bw + 1))
    for i in range(n):
        for j in range(max(0, i - bw), min(n, i + bw + 1)):
            band[i, j - i + bw] = K[i, j]
    _x, st = _solve(band, n, bw, A.SYSTEM_BAND_GENERAL, rhs)
    assert st == A.STRUT_SINGULAR

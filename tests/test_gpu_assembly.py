"""Assembly of band and F_int, and the pivoted band solve, at the sizes where their variants change:
2D rows (eight lanes a row, 32 rows a pass), 3D contribution lists (short, and longer than 24 for a
warp), window heights of the pivoted factorisation (32, 58, 64 rows) and more unknowns than the 224
columns it holds at a time.

Bars: the state determination as in the other state-determination tests (1e-9 of the largest entry,
against the oracle); the solve against numpy's dense LU of the same band, residual below 1e-12 of
|K| |x| (a backward-stable elimination leaves a small multiple of n eps = 1e-13)."""
import numpy as np
import pytest

from strut_b200 import model as M
from strut_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _check(gpu_lib, oracle, cases, amp, seed):
    models = [M.Model(c) for c in cases]
    rng = np.random.default_rng(seed)
    us = [rng.normal(0.0, amp, m.num_free) for m in models]
    with gpu_lib.Analysis(models) as an:
        got = an.state_determination(us)
    for m, u, (f, band) in zip(models, us, got):
        f_ref, band_ref, _bw = oracle.state_determination(m, u)
        assert np.max(np.abs(f - f_ref)) <= 1e-9 * np.max(np.abs(f_ref))
        assert np.max(np.abs(band - band_ref)) <= 1e-9 * np.max(np.abs(band_ref))


@pytest.mark.parametrize("sizes", [[(1, 1)], [(4, 2), (1, 5)], [(11, 1), (3, 7)], [(12, 5)]])
def test_assembly_2d(gpu_lib, oracle, sizes):
    _check(gpu_lib, oracle, [W.rc_frame_case(stories=s, bays=b, steps=2, seed=s) for s, b in sizes], 1e-4, 3)


@pytest.mark.parametrize("sizes,diaphragm", [([(1, 1)], False), ([(1, 1), (2, 2)], True), ([(2, 3)], True)])
def test_assembly_3d(gpu_lib, oracle, sizes, diaphragm):
    cases = [W.rc_frame3d_case(stories=s, bays_x=b, bays_y=1, steps=2, element="dispBeamColumn3d",
                               diaphragm=diaphragm, seed=s) for s, b in sizes]
    _check(gpu_lib, oracle, cases, 2e-4, 4)


@pytest.mark.parametrize("stories,bx,by", [(2, 1, 1), (3, 2, 2), (4, 3, 3), (3, 4, 3), (2, 8, 1), (10, 2, 2)])
def test_pivoted_solve(gpu_lib, stories, bx, by):
    case = W.rc_frame3d_case(stories=stories, bays_x=bx, bays_y=by, steps=2, element="dispBeamColumn3d",
                             diaphragm=True, seed=stories)
    m = M.Model(case)
    n = m.num_free
    rng = np.random.default_rng(n)
    with gpu_lib.Analysis([m]) as an:
        (_f, band), = an.state_determination([rng.normal(0.0, 1e-4, n)])
        bw, _rw = an.band_info(0)
        K = np.zeros((n, n))
        for i in range(n):
            for j in range(max(0, i - bw), min(n, i + bw + 1)):
                K[i, j] = band[i, j - i + bw]
        for k in range(2):  # the first solve finds the row swap, the second goes straight to pivoting
            rhs = rng.standard_normal(n)
            (x,) = an.factor_solve([rhs])
            assert np.linalg.norm(K @ x - rhs) <= 1e-12 * np.linalg.norm(K) * np.linalg.norm(x)

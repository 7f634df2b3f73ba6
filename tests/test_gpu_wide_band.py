"""The global-memory band LU on both sides of its narrow variants' limits (half bands 96 and 160: 128
and 192 threads, one per panel row; beyond them 384) and with a last panel that is not full, against
numpy's dense solve of the exported band.  Both solves are backward stable, so they differ by a small
multiple of eps times the condition number, below 1e6 for these frames: 1e-9 of the largest entry."""
import numpy as np
import pytest

from strut_b200 import model as M
from strut_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bays_x,bays_y,stories,bw", [(3, 2, 3, 77), (4, 2, 2, 95), (4, 2, 3, 95), (3, 3, 2, 101),
                                                      (3, 3, 3, 101), (4, 4, 2, 155), (5, 4, 2, 185)])
def test_exported_band_solve(gpu_lib, bays_x, bays_y, stories, bw):
    case = W.rc_frame3d_case(stories=stories, bays_x=bays_x, bays_y=bays_y, steps=4, element="dispBeamColumn3d",
                             seed=41, pga_g=0.4)
    m = M.Model(case)
    n = m.num_free
    u = np.random.default_rng(11).normal(0.0, 2e-4, n)
    rhs = np.random.default_rng(12).normal(size=n)
    with gpu_lib.Analysis([m]) as an:
        got_bw, rw = an.band_info(0)
        assert got_bw == bw and n * rw * 8 > 220 * 1024
        (_f, band), = an.state_determination([u])
        du, = an.factor_solve([rhs])
    K = np.zeros((n, n))
    for i in range(n):
        j = np.arange(max(0, i - bw), min(n, i + bw + 1))
        K[i, j] = band[i, j - i + bw]
    ref = np.linalg.solve(K, rhs)
    assert np.max(np.abs(du - ref)) <= 1e-9 * np.max(np.abs(ref))

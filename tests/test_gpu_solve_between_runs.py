"""A run gives the same bits whether or not factor_solve was called before it or between its steps, also where
the solved system needs row interchanges and the run's own do not."""
import numpy as np
import pytest

from strut_b200 import model as M
from strut_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _needs_interchange(band, bw):
    n = band.shape[0]
    K = np.zeros((n, n))
    for i in range(n):
        j = np.arange(max(0, i - bw), min(n, i + bw + 1))
        K[i, j] = band[i, j - i + bw]
    for k in range(n - 1):
        if np.any(np.abs(K[k + 1:, k]) > abs(K[k, k])):
            return True
        K[k + 1:, k:] -= np.outer(K[k + 1:, k] / K[k, k], K[k, k:])
    return False


@pytest.mark.parametrize("diaphragm,seed", [(False, 2), (True, 4)])
def test_factor_solve_leaves_the_run_alone(gpu_lib, diaphragm, seed):
    def model():
        return M.Model(W.rc_frame3d_case(stories=1, bays_x=1, bays_y=1, steps=20, diaphragm=diaphragm))

    n = model().num_free
    u = np.random.default_rng(seed).normal(0.0, 4e-3, n)  # far beyond yield
    rhs = np.random.default_rng(2).normal(size=n)
    out, solved = [], []
    for solve in (False, True):
        with gpu_lib.Analysis([model()]) as an:
            for _ in range(2):
                done = an.state(0)[0]
                (_f, band), = an.state_determination([u])
                if solve:
                    assert _needs_interchange(band, an.band_info(0)[0])
                    solved += an.factor_solve([rhs]) + an.factor_solve([rhs])
                an.state_determination([done])
                an.run(10)
            out.append(an.history(0))
    assert all(np.array_equal(a, b) for a, b in zip(*out))
    assert np.array_equal(solved[0], solved[1]) and np.array_equal(solved[2], solved[3])

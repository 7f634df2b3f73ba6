"""Systems of frames with entries of 2^500 and more, or infinities, in the instances' own kernel: the solve of an
exported band against IEEE divisions, and a run with a mass that large against the oracle (1e-7 of peak,
the same iteration counts)."""
import numpy as np
import pytest

from strut_b200 import model as M
from strut_b200 import workloads as W
from tests.test_gpu_band_special import _ieee_solve
from tests.test_gpu_records import compare_histories

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("system", ["BandGeneral", "BandSPD"])
@pytest.mark.parametrize("stories,bays", [(2, 2), (3, 3), (5, 5), (3, 7)])  # half bands 11, 14, 20, 26
@pytest.mark.parametrize("value", [-np.inf, 1e160])
def test_factor_solve(gpu_lib, system, stories, bays, value):
    case = W.rc_frame_case(stories=stories, bays=bays, steps=2, seed=2)
    case["analysis"]["system"] = system
    m = M.Model(case)
    n = m.num_free
    rhs = np.random.default_rng(n).normal(size=n)
    rhs[n // 2] = value
    with gpu_lib.Analysis([m]) as an:
        (_f, band), = an.state_determination([np.zeros(n)])
        bw, _rw = an.band_info(0)
        x, = an.factor_solve([rhs])
    K = np.zeros((n, n))
    for i in range(n):
        for j in range(max(0, i - bw), min(n, i + bw + 1)):
            K[i, j] = band[max(i, j), abs(i - j)] if system == "BandSPD" else band[i, j - i + bw]
    want = _ieee_solve(K, bw, rhs, system == "BandSPD")
    assert np.array_equal(np.isnan(x), np.isnan(want))
    assert np.array_equal(np.where(np.isinf(x), x, 0.0), np.where(np.isinf(want), want, 0.0))
    ok = np.isfinite(want)
    if ok.any():  # both backward stable, condition numbers below 1e6: n eps 1e6 = 5e-9 at most
        assert np.max(np.abs(x[ok] - want[ok])) <= 5e-9 * np.max(np.abs(want[ok]))


def test_run_with_a_huge_mass(gpu_lib, oracle):
    steps = 30
    case = W.rc_frame_case(stories=3, bays=2, steps=steps, seed=4)
    case["masses"][0]["value"] = 1e160
    m = M.Model(case)
    with gpu_lib.Analysis([m]) as an:
        an.run(steps)
        got = an.history(0)
    *want, rc, failed = oracle.run_transient(m, steps)
    assert rc == 0, f"oracle failed at step {failed}"
    worst_d, worst_e, n_diff = compare_histories(*got, *want)
    assert worst_d <= 1e-7 and worst_e <= 1e-7 and n_diff == 0

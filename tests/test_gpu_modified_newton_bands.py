"""ModifiedNewton keeps the step's factors, so the band LU stores its multipliers in the column that its
other lanes read: every row split of that LU (half bands 11, 14, 20, 23, 35) over steps of several
iterations, histories within 1e-7 of peak of the oracle and the same iteration counts."""
import pytest

from strut_b200 import model as M
from strut_b200 import workloads as W
from tests.test_gpu_records import compare_histories

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bays", [2, 3, 5, 6, 10])
def test_kept_factors(gpu_lib, oracle, bays):
    steps = 40
    case = W.rc_frame_case(stories=2, bays=bays, steps=steps, seed=bays, pga_g=0.6)
    case["analysis"]["algorithm"] = "ModifiedNewton"
    case["analysis"]["max_iters"] = 60
    m = M.Model(case)
    with gpu_lib.Analysis([m]) as an:
        assert an.band_info(0)[0] == 3 * (bays + 1) + 2
        st = an.run(steps)
        gd, ge, gi = an.history(0)
    assert st.factorizations == steps and st.global_newton_iterations > 2 * steps
    rd, re, ri, rc, failed = oracle.run_transient(m, steps)
    assert rc == 0, f"oracle failed at step {failed}"
    worst_d, worst_e, n_diff = compare_histories(gd, ge, gi, rd, re, ri)
    assert worst_d <= 1e-7 and worst_e <= 1e-7, (worst_d, worst_e)
    assert n_diff == 0

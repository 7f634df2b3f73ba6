"""3D frames whose half band is beyond what the row and pivoted factorisations hold (62 and 63) and whose band
still fits in shared memory: the general elimination, and the dense restart where a row interchange is
needed (and the last half band of the pivoted one).  Histories 1e-7 of peak against the oracle, with
its iteration counts."""
import pytest

from strut_b200 import model as M
from strut_b200 import workloads as W
from tests.test_gpu_records import compare_histories

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stories,bx,by,diaphragm,bw", [(2, 3, 2, False, 77), (2, 5, 2, True, 62),
                                                         (2, 4, 3, True, 68), (2, 4, 4, True, 83)])
def test_run_against_the_oracle(gpu_lib, oracle, stories, bx, by, diaphragm, bw):
    steps = 20
    m = M.Model(W.rc_frame3d_case(stories=stories, bays_x=bx, bays_y=by, steps=steps, diaphragm=diaphragm,
                                  element="dispBeamColumn3d", seed=7))
    n = m.num_free
    with gpu_lib.Analysis([m]) as an:
        got_bw, rw = an.band_info(0)
        assert got_bw == bw and (n * rw + 6 * n) * 8 <= 220 * 1024
        an.run(steps)
        got = an.history(0)
    *want, rc, failed = oracle.run_transient(m, steps)
    assert rc == 0, f"oracle failed at step {failed}"
    worst_d, worst_e, n_diff = compare_histories(*got, *want)
    assert worst_d <= 1e-7 and worst_e <= 1e-7 and n_diff == 0

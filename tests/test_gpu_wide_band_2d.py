"""2D frames whose band does not fit in shared memory (beyond 220 KiB with its vectors): assembly, wide
factorisation and substitution, alone and in one handle with a frame whose band does fit.  Half bands 35
and 32 fill the factorisation's 32-column panels, 20 gives panels of 20 columns.

Bars as elsewhere: the state determination 1e-9 of the largest entry against the oracle; the solve
against numpy's dense solve of the exported band, 1e-11 of the largest entry (both backward stable,
condition numbers of 34: n eps 34 = 4e-12 at most); histories 1e-7 of peak with the oracle's iteration counts."""
import numpy as np
import pytest

from strut_b200 import model as M
from strut_b200 import workloads as W
from tests.test_gpu_records import compare_histories

pytestmark = pytest.mark.gpu

SIZES = [(12, 10, 35), (14, 9, 32), (34, 5, 20)]


def _model(stories, bays, steps, **kw):
    return M.Model(W.rc_frame_case(stories=stories, bays=bays, steps=steps, seed=stories, **kw))


def _dense(band, bw):
    n = band.shape[0]
    K = np.zeros((n, n))
    for i in range(n):
        j = np.arange(max(0, i - bw), min(n, i + bw + 1))
        K[i, j] = band[i, j - i + bw]
    return K


@pytest.mark.parametrize("stories,bays,bw", SIZES)
def test_state_determination_and_solve(gpu_lib, oracle, stories, bays, bw):
    m = _model(stories, bays, 2)
    n = m.num_free
    u = np.random.default_rng(5).normal(0.0, 1e-4, n)
    rhs = np.random.default_rng(6).normal(size=n)
    with gpu_lib.Analysis([m]) as an:
        got_bw, rw = an.band_info(0)
        assert got_bw == bw and (n * rw + 6 * n) * 8 > 220 * 1024
        (f, band), = an.state_determination([u])
        du, = an.factor_solve([rhs])
    f_ref, band_ref, _bw = oracle.state_determination(m, u)
    assert np.max(np.abs(f - f_ref)) <= 1e-9 * np.max(np.abs(f_ref))
    assert np.max(np.abs(band - band_ref)) <= 1e-9 * np.max(np.abs(band_ref))
    ref = np.linalg.solve(_dense(band, bw), rhs)
    assert np.max(np.abs(du - ref)) <= 1e-11 * np.max(np.abs(ref))


@pytest.mark.parametrize("stories,bays,bw", SIZES)
def test_run_against_the_oracle(gpu_lib, oracle, stories, bays, bw):
    steps = 60
    m = _model(stories, bays, steps)
    with gpu_lib.Analysis([m]) as an:
        an.run(steps)
        gd, ge, gi = an.history(0)
    rd, re, ri, rc, failed = oracle.run_transient(m, steps)
    assert rc == 0, f"oracle failed at step {failed}"
    worst_d, worst_e, n_diff = compare_histories(gd, ge, gi, rd, re, ri)
    assert worst_d <= 1e-7 and worst_e <= 1e-7, (worst_d, worst_e)
    assert n_diff == 0


def test_wide_and_narrow_in_one_handle(gpu_lib):
    """Each frame's history is its own run's, bit for bit."""
    steps = 20
    models = [_model(3, 3, steps), _model(12, 10, steps), _model(2, 4, steps, element="dispBeamColumn2d")]
    alone = []
    for m in models:
        with gpu_lib.Analysis([m]) as an:
            an.run(steps)
            alone.append(an.history(0))
    with gpu_lib.Analysis(models) as an:
        an.run(steps)
        for i, (d, e, it) in enumerate(alone):
            d2, e2, it2 = an.history(i)
            assert np.array_equal(it, it2) and np.array_equal(d, d2) and np.array_equal(e, e2)

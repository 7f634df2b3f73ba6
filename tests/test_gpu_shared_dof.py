"""2D elements whose two ends share a dof (one index at both ends, as the C ABI allows): every one of an
element's contributions to a slot and to F_int counts.  State determination against the oracle, 1e-9 of
the largest entry as in the other state-determination tests."""
import numpy as np
import pytest

from strut_b200 import model as M
from strut_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(1, 1)], [(3, 3), (2, 4)]])
@pytest.mark.parametrize("direction", [0, 1, 2])
def test_state_determination(gpu_lib, oracle, sizes, direction):
    models = [M.Model(W.rc_frame_case(stories=s, bays=b, steps=2, seed=s)) for s, b in sizes]
    for m in models:
        for e in m.elements:
            if all(m.free_index[e.dof[a]] >= 0 for a in (direction, 3 + direction)):
                e.dof[3 + direction] = e.dof[direction]
                break
        else:
            raise AssertionError("no element between free nodes")
    us = [np.random.default_rng(7).normal(0.0, 1e-4, m.num_free) for m in models]
    with gpu_lib.Analysis(models) as an:
        got = an.state_determination(us)
    for m, u, (f, band) in zip(models, us, got):
        f_ref, band_ref, _bw = oracle.state_determination(m, u)
        assert np.max(np.abs(f - f_ref)) <= 1e-9 * np.max(np.abs(f_ref))
        assert np.max(np.abs(band - band_ref)) <= 1e-9 * np.max(np.abs(band_ref))

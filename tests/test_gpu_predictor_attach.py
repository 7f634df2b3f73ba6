"""Attaching the learned predictor to an analysis: the caller's normalisation arrays are free on return."""
import ctypes as C

import numpy as np
import pytest
import torch

from strut_b200 import model as M
from strut_b200 import predictor as PR
from strut_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _model(steps=40):
    return PR.record_all_dofs(M.Model(W.rc_frame_case(stories=2, bays=2, steps=steps, seed=5)))


def test_page_locked_arrays_are_read_before_the_return(gpu_lib):
    """The analysis's stream has work in front of the copies, and the arrays change right after the call."""
    m = _model()
    pred = PR.LearnedPredictor(m.ndf, seed=1)
    mean = np.linspace(-1e-3, 1e-3, pred.n_in).astype(np.float32)
    scale = np.linspace(1.0, 2.0, pred.n_in).astype(np.float32)
    pinned = [torch.from_numpy(a.copy()).pin_memory() for a in (mean, scale, np.ones(m.ndf, np.float32))]
    fp = C.POINTER(C.c_float)
    with gpu_lib.Analysis([m]) as an:
        stream = torch.cuda.ExternalStream(gpu_lib.lib().strut_gpu_stream(an.h))
        with torch.cuda.stream(stream):
            torch.cuda._sleep(200_000_000)  # 0.1 s
        gpu_lib._check(gpu_lib.lib().strut_gpu_set_predictor(
            an.h, pred.net.m, *[C.cast(t.data_ptr(), fp) for t in pinned]), "set_predictor")
        for t in pinned:
            t.fill_(7.0)
        an._predictor = pred
        got = PR.device_features(an)  # of step 0: no increments yet
    X, _ = PR.raw_features(m, np.zeros((1, m.num_free)))
    assert np.allclose(got, (X[:got.shape[0]] - mean) * scale, rtol=1e-6, atol=1e-6)


def test_another_predictor_takes_the_place_of_the_first(gpu_lib):
    """Runs after the change are those of an analysis whose step loop is built anew for the second network
    (a change of launch shape that gives the same results makes it so)."""
    def predictor(seed):
        p = PR.LearnedPredictor(3, seed=seed)
        p.y_scale = np.full(3, 1e-4 * (seed + 1), np.float32)
        return p

    first, second = predictor(0), predictor(3)
    runs = []
    for rebuild in (False, True):
        with gpu_lib.Analysis([_model(60)], tuned=False) as an:
            first.attach(an)
            an.run(20)
            second.attach(an)
            if rebuild:
                an.set_tuning(element_threads=224)
            an.run(20)
            runs.append((*an.history(0), PR.stats(an)))
            PR.detach(an)
            an.run(20)
            runs[-1] += an.history(0)
    for a, b in zip(*runs):
        assert np.array_equal(a, b)

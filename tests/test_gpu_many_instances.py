"""3D batches of more instances than a grid has rows (65,535), and batches of very uneven instances: each
instance's history is the bits of its own run."""
import ctypes as C

import numpy as np
import pytest

from strut_b200 import _abi as A
from strut_b200 import model as M
from strut_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _cantilever(steps):
    """One column with a mass on it, four fibers in a section."""
    case = W.rc_frame3d_case(stories=1, bays_x=1, bays_y=1, steps=steps, nip=3, element="dispBeamColumn3d",
                             record_elements=())
    top = next(e for e in case["elements"] if e["id"] == 1)["nodes"][1]
    case["elements"] = case["elements"][:1]
    case["nodes"] = [n for n in case["nodes"] if n["id"] in case["elements"][0]["nodes"]]
    case["masses"] = [m for m in case["masses"] if m["node"] == top]
    case["recorders"][0]["nodes"] = [top]
    p = case["sections"][0]["params"]
    p["layers"] = []
    p["patches"] = [dict(p["patches"][0], num_subdiv_y=2, num_subdiv_z=2)]
    return case


def test_more_instances_than_grid_rows(gpu_lib):
    steps, n = 3, 65_600
    m = M.Model(_cantilever(steps))
    with gpu_lib.Analysis([m]) as an:
        an.run(steps)
        want, _e, iters = an.history(0)
    desc = m.desc()  # one description n times
    descs = (A.StrutModelDesc * n)(*([desc] * n))
    h = C.c_void_p()
    gpu_lib._check(gpu_lib.lib().strut_gpu_create(descs, n, -1, C.byref(h)), "create")
    an = gpu_lib.Analysis.__new__(gpu_lib.Analysis)
    an.models, an.h, an.steps_done = [m] * n, h, 0
    with an:
        an.run(steps)
        d, _e, it = an.history_all()
        assert not an.instance_status().any()
    assert np.abs(want).max() > 0.0
    assert np.array_equal(d.reshape(n, steps, -1), np.broadcast_to(want, (n, *want.shape)))
    assert np.array_equal(it.reshape(n, steps), np.broadcast_to(iters, (n, steps)))


def test_uneven_instances(gpu_lib):
    steps = 10
    models = [M.Model(_cantilever(steps)),
              M.Model(W.rc_frame3d_case(stories=3, bays_x=2, bays_y=2, steps=steps, diaphragm=True)),
              M.Model(_cantilever(steps))]
    alone = []
    for m in models:
        with gpu_lib.Analysis([m]) as an:
            an.run(steps)
            alone.append(an.history(0))
    with gpu_lib.Analysis(models) as an:
        an.run(steps)
        for i, ref in enumerate(alone):
            assert all(np.array_equal(a, b) for a, b in zip(an.history(i), ref))

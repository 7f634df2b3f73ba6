"""Several analyses or section batches alive at once: a smaller one made after a larger one leaves the larger
one's launches as they were, and threads that make, run and give back analyses side by side share the
pool of device memory.  Every run gives the bits of the same run alone."""
import threading

import numpy as np
import pytest
import torch

from strut_b200 import model as M
from strut_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _frame(stories, bays, steps=20):
    return M.Model(W.rc_frame_case(stories=stories, bays=bays, steps=steps, seed=stories))


def _alone(gpu_lib, size, steps):
    with gpu_lib.Analysis([_frame(*size)]) as an:
        an.run(steps)
        return an.history(0)


@pytest.mark.parametrize("large", [(12, 5), (34, 5)], ids=["shared", "wide"])
def test_larger_analysis_runs_after_a_smaller_was_made(gpu_lib, large):
    small = (12, 10) if large == (34, 5) else (2, 2)
    want = [_alone(gpu_lib, s, 20) for s in (large, small)]
    a = gpu_lib.Analysis([_frame(*large)])
    b = gpu_lib.Analysis([_frame(*small)])
    rhs = np.ones(a.models[0].num_free)
    a.state_determination([np.zeros_like(rhs)])
    assert np.isfinite(a.factor_solve([rhs])[0]).all()
    for an, ref in ((a, want[0]), (b, want[1])):
        an.run(20)
        assert all(np.array_equal(x, y) for x, y in zip(an.history(0), ref))
        an.close()


def test_larger_section_batch_evaluates_after_a_smaller_was_made(gpu_lib):
    case = W.rc_frame_case(stories=1, bays=1, steps=2)
    mats, nm, fibs, nf = M.section_fibers(case["sections"][0], case["materials"])
    few = 6
    n = 37
    ek = torch.linspace(-2e-3, 2e-3, 2 * n, dtype=torch.float64, device="cuda")
    out = []
    for alone in (True, False):
        a = gpu_lib.SectionBatch(mats, nm, fibs, nf, n)
        b = None if alone else gpu_lib.SectionBatch(mats, nm, fibs, few, n)
        resp = torch.zeros(n, 5, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        a.eval(ek.data_ptr(), resp.data_ptr())
        torch.cuda.synchronize()
        out.append(resp.cpu())
        a.close()
        if b:
            b.close()
    assert torch.equal(*out)


def test_threads_share_the_pool(gpu_lib):
    sizes = [(3, 3), (5, 2), (2, 4), (6, 1)]
    want = [_alone(gpu_lib, s, 20) for s in sizes]
    wrong = []

    def work(k):
        try:
            for _ in range(3):
                got = _alone(gpu_lib, sizes[k], 20)
                if not all(np.array_equal(x, y) for x, y in zip(got, want[k])):
                    wrong.append(k)
        except Exception as exc:  # a thread's failure fails the test
            wrong.append(repr(exc))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong

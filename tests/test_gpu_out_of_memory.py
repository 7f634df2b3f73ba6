"""An object too large for the device is refused with an error, and the next one is made and used as if nothing
had been asked."""
import numpy as np
import pytest
import torch

from strut_b200 import model as M
from strut_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_refused_batch_leaves_no_error_behind(gpu_lib):
    case = W.rc_frame_case(stories=1, bays=1, steps=5)
    mats, nm, fibs, nf = M.section_fibers(case["sections"][0], case["materials"])
    with pytest.raises(gpu_lib.StrutError):
        gpu_lib.SectionBatch(mats, nm, fibs, nf, 2_000_000_000)  # 11 TB of Concrete02 history
    ek = torch.zeros(6, dtype=torch.float64, device="cuda")
    resp = torch.zeros(3, 5, dtype=torch.float64, device="cuda")
    batch = gpu_lib.SectionBatch(mats, nm, fibs, nf, 3)
    batch.eval(ek.data_ptr(), resp.data_ptr())
    torch.cuda.synchronize()
    assert (resp[:, 2] > 0.0).all()
    batch.close()
    with pytest.raises(gpu_lib.StrutError):
        gpu_lib.SectionBatch(mats, nm, fibs, nf, 2_000_000_000)
    with gpu_lib.Analysis([M.Model(case)]) as an:
        an.run(5)
        assert np.isfinite(an.history(0)[0]).all()

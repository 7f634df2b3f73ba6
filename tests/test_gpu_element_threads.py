"""The default size of an element CTA: 640 threads for force-based elements of more than 960 fibers (148 a
section: seven points) where 320 would put no more elements in flight, else 320; the same bits as with
the sizes set by hand."""
import numpy as np
import pytest

from strut_b200 import model as M
from strut_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _frames(n, nip, element, steps=10):
    return [M.Model(W.rc_frame_case(stories=6, bays=3, steps=steps, nip=nip, element=element, seed=i, pga_g=1.5))
            for i in range(n)]


@pytest.mark.parametrize("n,nip,element,threads", [
    (1, 6, "forceBeamColumn2d", 320), (1, 7, "forceBeamColumn2d", 640), (1, 7, "dispBeamColumn2d", 320),
    (3, 7, "forceBeamColumn2d", 640),   # 126 elements
    (4, 7, "forceBeamColumn2d", 320),   # 168: more than the 148 SMs
    (4, 10, "forceBeamColumn2d", 640)])  # one CTA an SM with either size
def test_default(gpu_lib, n, nip, element, threads):
    out = []
    for by_hand in (None, 320, 640):
        with gpu_lib.Analysis(_frames(n, nip, element), tuned=False) as an:
            if by_hand:
                an.set_tuning(element_threads=by_hand)
            assert an.tuning().element_threads == (by_hand or threads)
            an.run(10, check=False)
            out.append(an.history_all())
    for other in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(out[0], other))

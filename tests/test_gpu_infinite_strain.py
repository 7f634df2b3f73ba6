"""Strain histories that run through infinities or strains whose quotients overflow, against the oracle's
divisions: NaN and infinities where it has them, finite values as in the other path tests (1e-9 of
the largest finite entry)."""
import numpy as np
import pytest

from strut_b200 import model as M
from tests.test_gpu_parity import MATS

pytestmark = pytest.mark.gpu

INF = np.inf
PATHS = {
    "tension": [1e-3, INF, 1e-3, -2e-3],
    "compression": [-1e-3, -INF, -1e-3, 5e-4],
    "both": [1e-2, INF, 0.0, -1e-2, -INF, 0.0, 1e-2],
    "huge": [1e-2, 1e306, 0.0, -1e306, 1e-2, -1e-2],
    "first": [INF, 1e-3, -1e-3],
}


@pytest.mark.parametrize("path", sorted(PATHS))
@pytest.mark.parametrize("mat", MATS, ids=[m["type"] + str(m["id"]) for m in MATS])
def test_material_path(gpu_lib, oracle, mat, path):
    m = M.uniaxial_material(mat)
    strains = np.array(PATHS[path])
    with np.errstate(all="ignore"):
        ref = oracle.material_path(m, strains)
    got = gpu_lib.material_path(m, strains)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert np.array_equal(np.where(np.isinf(got), got, 0.0), np.where(np.isinf(ref), ref, 0.0))
    ok = np.isfinite(ref)
    # 1e306 E0 is finite: such stresses are compared with themselves, the others with the largest of them
    big = ok & (np.abs(ref) > 1e200)
    np.testing.assert_allclose(got[big], ref[big], rtol=1e-9)
    ok &= ~big
    np.testing.assert_allclose(got[ok], ref[ok], rtol=1e-9, atol=1e-9 * np.abs(ref[ok]).max(initial=0.0))

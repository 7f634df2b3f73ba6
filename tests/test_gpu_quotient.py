"""The quotient that the band LU and the constitutive laws take instead of an FP64 division, against
numpy's (correctly rounded) division, seen through a band solve of 2 x 2 blocks

    [a 0; b 1] x = [1; 0]   with   x = [1 / a; -(b / a)].

The quotient v r corrected with the exact residual v - q d has an error of half an ulp plus a
rounding of the correction (at most 2^-50 ulp, as r is within two ulps of 1 / d), so it is the
correctly rounded value or, next to a tie, its neighbour: one ulp is the bound.  Divisors and
numerators cover 24 decades with random mantissas, powers of two, and zero numerators."""
import numpy as np
import pytest

from strut_b200 import _abi as A
from tests.test_gpu_band_solve import _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(16))
@pytest.mark.parametrize("bw", [1, 13])  # one warp a row set; a CTA
def test_quotient_within_one_ulp(bw, seed):
    rng = np.random.default_rng(seed)
    nb = 250
    a = rng.uniform(1.0, 2.0, nb) * 2.0 ** rng.integers(-38, 41, nb) * rng.choice([-1.0, 1.0], nb)
    b = a * rng.uniform(-1.0, 1.0, nb) * 2.0 ** -rng.integers(0, 40, nb)
    a[:8] = 2.0 ** np.arange(-4, 4)
    b[8:16] = 0.0
    n = 2 * nb
    band = np.zeros((n, 2 * bw + 1))
    band[0::2, bw] = a
    band[1::2, bw] = 1.0
    band[1::2, bw - 1] = b
    rhs = np.zeros(n)
    rhs[0::2] = 1.0
    x, st = _solve(band, n, bw, A.SYSTEM_BAND_GENERAL, rhs)
    assert st == 0
    for got, want in ((x[0::2], 1.0 / a), (x[1::2], -(b / a))):
        assert np.all(np.abs(got - want) <= np.spacing(np.abs(want)))
    assert np.all(x[1::2][8:16] == 0.0)

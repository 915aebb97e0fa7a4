"""Cell volumes and masses beyond the whole range of the branch-free division
(2^-240..2^240, lare_div.cuh): its fall-back gives the oracle's bits, as do
scales that it takes on the straight path."""
import pytest

from tests import test_gpu_scales as scales

pytestmark = pytest.mark.gpu


def _thinnest_density(F, rng):
    F[0][...] *= 1e-73  # mass per cell below 2^-240
    for f in (9, 10, 11):
        F[f] *= 1e-40


@pytest.mark.parametrize("case,n,scale,change", [
    ("rf", (9, 8, 26), 1e26, None),   # volumes above 2^239
    ("ot", (12, 10, 4), 1e-26, None),  # ... below 2^-240
    ("rf", (9, 10, 11), 1e20, None),  # ... 2^190: the straight path
    ("rf", (9, 10, 11), 1.0, _thinnest_density),
])
@pytest.mark.parametrize("batched", [False, True])
def test_far_scales_match_oracle(case, n, scale, change, batched, oracle_lib):
    scales.test_fallback_matches_checker(case, n, scale, change, batched, oracle_lib)

"""The fraction tree around the height (2^19 inputs) where its first build launch stops after five
levels, against the oracle byte for byte."""
import pytest

from tests import test_gpu_logup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [15, 18, 19, 20])
def test_frac_sum_build_heights(lgs, orc, k):
    test_gpu_logup.test_frac_sum_matches_oracle(lgs, orc, k)

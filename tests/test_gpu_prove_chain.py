"""The Basefold chain's launches at the edges of their ranges, whole roots and proofs against the
oracle byte for byte: the shortest codewords, the lengths around which one, two and three levels
fold in a launch, transforms on columns, with too few columns for that, and on rows."""
import pytest

from tests.test_gpu_basefold import _run

pytestmark = pytest.mark.gpu


# 2^(n - li + rate) code values of 2^li (twice that in the extension) columns
@pytest.mark.parametrize("is_ef,n,code_rate,li", [
    (False, 2, 1, 1), (True, 2, 1, 0), (False, 7, 3, 6), (True, 9, 1, 4), (False, 9, 2, 0),
    (True, 10, 1, 0), (False, 11, 1, 1), (False, 12, 1, 1), (False, 13, 2, 2), (True, 13, 1, 0),
    (False, 16, 1, 3), (False, 17, 2, 6)])
def test_basefold_chain_matches_oracle(lgs, orc, is_ef, n, code_rate, li):
    r = _run(orc, is_ef, n, code_rate, li, seed=300 + 40 * n + 7 * li + code_rate)
    assert r["commit"].root == r["cm"].root
    assert r["proof"].data == r["want"]

"""Basefold proofs at every number of columns, whose level-0 combination gives a row to one to eight
lanes: the fewest rows, less than a CTA of them, and more than the grid takes at once.  Byte for byte
against the oracle."""
import pytest

from tests.test_gpu_basefold import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("is_ef", [False, True])
@pytest.mark.parametrize("li", range(7))
@pytest.mark.parametrize("rows", [2, 128])
def test_few_rows(lgs, orc, is_ef, li, rows):
    r = _run(orc, is_ef, li + rows.bit_length() - 1, 1, li, seed=400 + 10 * li + rows)
    assert r["proof"].data == r["want"]


@pytest.mark.parametrize("is_ef,li,n,code_rate", [(False, 0, 17, 2), (True, 1, 17, 2),
                                                  (False, 3, 18, 4), (False, 4, 18, 3),
                                                  (True, 5, 18, 3)])
def test_many_rows(lgs, orc, is_ef, li, n, code_rate):
    r = _run(orc, is_ef, n, code_rate, li, seed=500 + n + li)
    assert r["proof"].data == r["want"]

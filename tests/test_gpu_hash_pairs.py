"""Subset-sum hash on CTA pairs at the edges of its work units, against the oracle (exact)."""
import numpy as np
import pytest

from ligesis_b200 import rng
from ligesis_b200._lib import Context, check, load, ptr64
from tests.helpers import P

pytestmark = pytest.mark.gpu


# m: one chunk of two rows, odd rows, a half-filled last stage (two chunks), K splits that do not
# divide the chunks; cols: one tile, a ragged last tile; hash_ctas: one pair (from 1 and from 2),
# odd counts, all of them
@pytest.mark.parametrize("m,cols,hash_ctas", [
    (1, 256, 0), (2, 200, 1), (5, 700, 2), (6, 513, 3), (7, 5 * 256, 5), (8, 256, 148),
    (33, 3 * 256, 7), (130, 512, 0), (259, 256, 9), (601, 3 * 256 + 1, 0)])
def test_hash_pairs_match_oracle(lgs, orc, m, cols, hash_ctas):
    A = rng.field_elements(2300 + m, 32 * 64 * m).reshape(32, 64 * m)
    cw = rng.field_elements(3300 + m, m * cols).reshape(m, cols)
    cw[0, 0], cw[m - 1, cols - 1] = P - 1, 0
    ctx = Context(0)
    ctx.tune(hash_ctas=hash_ctas)
    got = np.zeros((32, cols), dtype=np.uint64)
    check(load().lgs_subset_sum_hash(ctx.handle, ptr64(A), m, ptr64(cw), cols, ptr64(got)))
    assert np.array_equal(got, orc.hash_columns(A, cw))

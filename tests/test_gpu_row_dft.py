"""The row transforms (2^12 .. 2^20) where their splits change: every final pass, rows full and
padded from N/2, N/4 and N/8 values, 1, 2 and 4 columns per CTA with a ragged last CTA, and inputs
at the ends of the 24-bit limbs and beyond p.  Against the oracle's DFT, exact."""
import numpy as np
import pytest

import ligesis_b200 as L
from ligesis_b200 import rng
from tests.helpers import P

pytestmark = pytest.mark.gpu


def canon(c):
    return np.where(c >= np.uint64(P), c - np.uint64(P), c)


def check(orc, c, log_size, rows):
    got = L.dft(c, log_size)
    for b in rows:
        assert np.array_equal(got[b], orc.dft_bf(canon(c[b]), 1 << log_size)), b


@pytest.mark.parametrize("log_size", range(12, 21))
@pytest.mark.parametrize("pad", [0, 1, 2, 3])
def test_every_size_and_padding(lgs, orc, log_size, pad):
    c = rng.field_elements(40 * log_size + pad, 2 << (log_size - pad)).reshape(2, -1)
    check(orc, c, log_size, (0, 1))


@pytest.mark.parametrize("log_size,rows", [(12, 1), (12, 297), (12, 593), (13, 1), (13, 149),
                                           (13, 297), (14, 75), (14, 149), (15, 37)])
def test_columns_per_cta(lgs, orc, log_size, rows):
    # 592 and more columns run four to a CTA, 296 and more two, fewer one (2^13: two)
    c = rng.field_elements(7000 + rows, rows << (log_size - 1)).reshape(rows, -1)
    check(orc, c, log_size, sorted({0, rows // 2, rows - 1}))


@pytest.mark.parametrize("log_size", [12, 13, 15, 16, 17, 18, 19, 20])
def test_limb_edges(lgs, orc, log_size):
    n = 1 << log_size
    edge = np.array([(1 << 64) - 1, 0, (1 << 24) - 1, ((1 << 24) - 1) << 24, 0xFFFF << 48, P, P - 1,
                     P + 1, 1 << 63], dtype=np.uint64)
    c = np.stack([np.full(n, (1 << 64) - 1, dtype=np.uint64), edge[np.arange(n) % edge.size],
                  edge[(rng.ints(log_size, n) % np.uint64(edge.size)).astype(np.int64)]])
    check(orc, c, log_size, (0, 1, 2))

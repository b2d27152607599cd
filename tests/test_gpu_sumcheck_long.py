"""Sumchecks of one and two factors past the length from which their passes are streamed: one to
three streamed passes before two of tiles, odd and even lengths, and the last length that is not
streamed.  Exact, against the oracle."""
import numpy as np
import pytest

import ligesis_b200 as L
from ligesis_b200 import rng

pytestmark = pytest.mark.gpu


def _inputs(d, k):
    g = np.random.default_rng(100 * d + k)
    polys = [g.integers(0, rng.P, size=(1 << k, 2), dtype=np.uint64) for _ in range(d)]
    for p in polys:
        p[:4], p[-4:] = 0, rng.P - 1
    return polys, rng.ext_elements(810 + k, k)


@pytest.mark.parametrize("d,k", [(1, 22), (1, 23), (1, 24), (1, 25), (1, 27), (2, 22), (2, 23),
                                 (2, 24)])
def test_streamed_passes(lgs, orc, d, k):
    polys, ch = _inputs(d, k)
    ctx = L.Context(0)  # its arena holds the factors and goes with it
    try:
        rounds, finals = L.sumcheck_prove(polys, ch, ctx)
    finally:
        ctx.close()
    want_r, want_f, _ = orc.sumcheck_prove(polys, ch)
    assert np.array_equal(rounds, want_r) and np.array_equal(finals, want_f)

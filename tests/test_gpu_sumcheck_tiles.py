"""The tiled sumcheck where its plan changes: fewer pairs than a warp, one tile, the smallest and
longest single pass, two passes, and few CTAs that walk several tiles each.  Exact, against the
oracle."""
import numpy as np
import pytest

import ligesis_b200 as L
from ligesis_b200 import rng

pytestmark = pytest.mark.gpu

EDGE = np.array([0, 1, rng.P - 1, (1 << 22) - 1,
                 1 << 22, 1 << 44, 0xFFFFFFFF, 1 << 32], dtype=np.uint64)


@pytest.mark.parametrize("d", [1, 2, 3])
@pytest.mark.parametrize("k", [1, 2, 5, 6, 7, 10, 11, 18, 19])
def test_pass_plans(lgs, orc, d, k):
    polys = [rng.ext_elements(610 + 10 * d + j, 1 << k) for j in range(d)]
    polys[0][::5, 1] = EDGE[np.arange(polys[0][::5].shape[0]) % EDGE.size]
    ch = rng.ext_elements(710 + k, k)
    want_r, want_f, _ = orc.sumcheck_prove(polys, ch)
    rounds, finals = L.sumcheck_prove(polys, ch)
    assert np.array_equal(rounds, want_r)
    assert np.array_equal(finals, want_f)


@pytest.mark.parametrize("blocks", [1, 3, 16])
def test_few_ctas(lgs, orc, blocks):
    k, ctx = 15, L.Context(0)
    polys = [rng.ext_elements(650 + j, 1 << k) for j in range(2)]
    ch = rng.ext_elements(750, k)
    ctx.tune(sumcheck_blocks=blocks)
    try:
        rounds, finals = L.sumcheck_prove(polys, ch, ctx)
    finally:
        ctx.close()
    want_r, want_f, _ = orc.sumcheck_prove(polys, ch)
    assert np.array_equal(rounds, want_r) and np.array_equal(finals, want_f)

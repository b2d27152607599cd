"""The device field operations at the edges of their carries and corrections, through the smallest
calls that run them: a 2-point DFT (one sum, one difference) and a one-variable evaluation
(v0 + r (v1 - v0) over F_{p^2}), against Python's integers.  Exact."""
import itertools

import numpy as np
import pytest

import ligesis_b200 as L
from ligesis_b200 import field as fld

pytestmark = pytest.mark.gpu

P = fld.P
EDGES = [0, 1, 2, 7, 2**31, 2**32 - 2, 2**32 - 1, 2**32, 2**32 + 1, 2**33 - 1, 2**63 - 1, 2**63,
         P - 2**32, P - 2**32 + 1, P - 7, P - 2, P - 1]


def test_sum_and_difference_edges():
    pairs = np.array(list(itertools.product(EDGES, EDGES)), dtype=np.uint64)
    out = L.dft(pairs, 1)
    for (a, b), (s, d) in zip(pairs.tolist(), out.tolist()):
        assert (s, d) == ((a + b) % P, (a - b) % P)


@pytest.mark.parametrize("c1", [0, 1, 2**32 - 1, P - 1])
def test_extension_product_edges(c1):
    ctx = L.Context.default(0)
    for v, r in itertools.product(EDGES, EDGES):
        v0, v1, pt = (c1, v), (v, c1), (r, (v + c1) % P)
        want = fld.ef_add(v0, fld.ef_mul(pt, fld.ef_sub(v1, v0)))
        assert L.MlPoly([list(v0), list(v1)]).eval([pt], ctx) == want

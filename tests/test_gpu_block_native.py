"""The block's native call against the oracle: odd and single-row shapes, values that send it back
to the layers one by one, and the errors they report."""
import numpy as np
import pytest

import ligesis_b200 as L
from ligesis_b200 import proofsys as ps
from ligesis_b200._lib import Context

pytestmark = pytest.mark.gpu


def _cfg(n, d, heads, hidden):
    return {**ps.GPT2_31, "n_seq": n, "d_model": d, "n_head": heads, "mlp_hidden": hidden}


def _same(got, want):
    assert tuple(got) == ps.BLOCK_FIELDS
    for k in ps.BLOCK_FIELDS:
        assert got[k].dtype == np.int64 and np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("n,d,heads,hidden", [(1, 64, 1, 64), (2, 33, 3, 65), (31, 96, 6, 127),
                                              (33, 64, 4, 130), (70, 40, 5, 48)])
def test_native_block_matches_oracle(lgs, orc, n, d, heads, hidden):
    cfg = _cfg(n, d, heads, hidden)
    x, w, el, gl = ps.synthetic_block(3 + n, cfg)
    got = ps._block_on_device(x, w, el, gl, cfg, Context.default())
    _same(got, orc.block_witness(x, w, el, gl, cfg))


def test_block_outside_the_encodings(lgs, orc):
    cfg = _cfg(5, 64, 4, 96)
    x, w, el, gl = ps.synthetic_block(8, cfg)
    w["attn_w"][3, 5] = 1 << 16  # needs three limbs
    assert ps._block_on_device(x, w, el, gl, cfg, Context.default()) is None
    _same(ps.block_witness(x, w, el, gl, cfg), orc.block_witness(x, w, el, gl, cfg))


def test_block_errors_are_the_layers(lgs):
    cfg = _cfg(5, 64, 4, 96)
    x, w, el, gl = ps.synthetic_block(9, cfg)
    with pytest.raises(L.ShapeError, match="lookup gather"):
        ps.block_witness(x, w, el, gl[:8], cfg)
    with pytest.raises(ValueError, match="inner dimensions"):
        ps.block_witness(x, {**w, "attn_w": w["attn_w"][:-1]}, el, gl, cfg)

"""A block whose linear layers have no bias runs layer by layer.  The CPU test looks at the route
alone, the GPU test at the results."""
import numpy as np
import pytest

from ligesis_b200 import proofsys as ps

CFG = {**ps.GPT2_31, "n_seq": 5, "d_model": 24, "n_head": 3, "mlp_hidden": 40}
BIASES = ("attn_b", "attn_proj_b", "fc_b", "fproj_b")


def _without(w, names):
    return {k: None if k in names else v for k, v in w.items()}


@pytest.mark.parametrize("names", [(b,) for b in BIASES] + [BIASES])
def test_block_without_biases_is_left_to_the_layers(names):
    x, w, el, gl = ps.synthetic_block(5, CFG)
    assert ps._block_on_device(x, _without(w, names), el, gl, CFG, None) is None


@pytest.mark.gpu
@pytest.mark.parametrize("names", [("fc_b",), BIASES])
def test_block_without_biases_matches_oracle(lgs, orc, names):
    x, w, el, gl = ps.synthetic_block(6, CFG)
    zero = {k: np.zeros_like(v) if k in names else v for k, v in w.items()}
    want = orc.block_witness(x, zero, el, gl, CFG)
    got = ps.block_witness(x, _without(w, names), el, gl, CFG)
    for k in ps.BLOCK_FIELDS:
        assert np.array_equal(got[k], want[k]), k

"""The forms of a block's arguments: linear layers without a bias, which run layer by layer (the CPU
test looks at the route alone), and scales that are not Python ints."""
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


@pytest.mark.gpu
@pytest.mark.parametrize("as_type", [float, np.int64, np.float64])
def test_block_scale_of_any_number_type(lgs, orc, as_type):
    x, w, el, gl = ps.synthetic_block(7, CFG)
    want = orc.block_witness(x, w, el, gl, CFG)
    cfg = {**CFG, "scale": as_type(CFG["scale"]), "max_v": as_type(CFG["max_v"])}
    got = ps.block_witness(x, w, el, gl, cfg)
    for k in ps.BLOCK_FIELDS:
        assert np.array_equal(got[k], want[k]), k

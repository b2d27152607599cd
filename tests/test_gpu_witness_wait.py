"""The linear witness' bounded waits when they run out (a budget of one cycle, as
tests/test_gpu_bounded_wait.py does for the hash): the persistent tensor-core kernel and the block
report DeviceTimeout, also where results leave the i64 range in the same call, and afterwards the
same context gives the oracle's results and reports a range error as one.  (The kernel of a CTA per
unit looks at its budget only after a suspension that its short waits never outlast.)"""
import numpy as np
import pytest

import ligesis_b200 as L
from ligesis_b200 import proofsys as ps

pytestmark = pytest.mark.gpu

TOP = (1 << 63) - 1


def _rand(seed, shape, bound):
    return np.random.default_rng(seed).integers(-bound, bound, size=shape, dtype=np.int64)


@pytest.mark.parametrize("wt", [False, True])
def test_linear_wait_gives_up_and_the_context_stays_usable(lgs, orc, wt):
    rows, inner, cols = 31, 2048, 1024
    x = _rand(1, (rows, inner), 1 << 21)
    w = _rand(2, (cols, inner) if wt else (inner, cols), 1 << 15)
    b = _rand(3, cols, 1 << 30)
    over = np.where(np.arange(cols) % 2, TOP, -TOP)  # Q + bias leaves i64 in every other column
    want = orc.linear_witness(x, w, b, 1 << 12, wt)
    ctx = L.Context(0)
    try:
        for bias in (b, over, b):
            ctx.set_wait_budget(1)
            with pytest.raises(L.DeviceTimeout, match="bounded device wait"):
                ps.linear_witness(x, w, bias, 1 << 12, wt, ctx)
            ctx.set_wait_budget(0)
            for got, exp in zip(ps.linear_witness(x, w, b, 1 << 12, wt, ctx), want):
                assert np.array_equal(got, exp)
            with pytest.raises(L.ShapeError, match="i64 range"):
                ps.linear_witness(x, w, over, 1 << 12, wt, ctx)
    finally:
        ctx.close()


def test_block_wait_gives_up_and_the_context_stays_usable(lgs, orc):
    x, w, el, gl = ps.synthetic_block(21, ps.GPT2_31)
    want = orc.block_witness(x, w, el, gl, ps.GPT2_31)
    ctx = L.Context(0)
    try:
        for _ in range(2):
            ctx.set_wait_budget(1)
            with pytest.raises(L.DeviceTimeout, match="bounded device wait"):
                ps.block_witness(x, w, el, gl, ps.GPT2_31, ctx)
            ctx.set_wait_budget(0)
            got = ps._block_on_device(x, w, el, gl, ps.GPT2_31, ctx)
            for k in ps.BLOCK_FIELDS:
                assert np.array_equal(got[k], want[k]), k
    finally:
        ctx.close()

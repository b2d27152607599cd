"""A polynomial in page-locked memory, which the DMA engine reads after `Ligesis.commit` returns, lives
until the commit is done: the root read, or a prove returned."""
import gc
import weakref

import numpy as np
import pytest

import ligesis_b200 as L
from ligesis_b200 import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("by", ["root", "prove"])
def test_page_locked_values_outlive_the_caller(lgs, by):
    torch = pytest.importorskip("torch")
    log_m, log_n = 5, 14
    hash_ = L.SubsetSumHash(64 << log_m, a=rng.field_elements(1, 2048 << log_m).reshape(32, -1))
    pk, _ = L.Ligesis.setup_with_hash(log_m, log_n, hash_, L.Context.default(0))
    v = rng.field_elements(2, 1 << (log_m + log_n))
    want = L.Ligesis.commit(pk, L.MlPoly(v))[0].root
    pin = torch.empty(v.size, dtype=torch.int64, pin_memory=True)
    pin.numpy().view(np.uint64)[:] = v
    f = L.MlPoly(pin.numpy().view(np.uint64))
    assert f.evals.ctypes.data == pin.data_ptr()  # not a copy
    values = weakref.ref(f.evals)
    commit, data = L.Ligesis.commit(pk, f)
    del f, pin
    gc.collect()
    assert values() is not None
    if by == "prove":
        L.Ligesis.prove(pk, data, rng.ext_elements(3, log_m + log_n),
                        L.RandomOracle(rng.SeededRng(4), length=2048))
        assert values() is None
    assert commit.root == want and values() is None

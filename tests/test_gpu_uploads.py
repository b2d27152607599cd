"""Uploads of pageable arrays through the pinned ring: sources off 16-byte alignment, less than a
line, just around the ring's 8 MB chunks and the copy pool's 1 MB parts, against the device's own
result for the same values."""
import numpy as np
import pytest

import ligesis_b200 as L
from ligesis_b200 import rng

pytestmark = pytest.mark.gpu


def _unaligned(a, shift):
    b = np.empty(a.size + 8, dtype=np.uint64)
    s = (-(b.ctypes.data // 8) % 8 + shift) % 8  # `shift` words past a 64-byte line
    b[s:s + a.size] = a
    return b[s:s + a.size]


# Basefold stages n values in one piece: 2^1 .. 2^21 of them (16 bytes to two chunks)
@pytest.mark.parametrize("n,li,shift", [(1, 0, 1), (2, 0, 3), (5, 2, 7), (10, 6, 1), (17, 6, 5),
                                        (18, 6, 0), (20, 6, 1), (21, 6, 3)])
def test_staged_upload_any_alignment(lgs, orc, n, li, shift):
    v = rng.field_elements(70 + n, 1 << n)
    _, com = L.Basefold.commit_base_on_domain(L.MlPoly(_unaligned(v, shift)), 1, li)
    assert com.root == orc.BasefoldCommitment(v, False, 1, li).root


# whole rows in blocks of 8 MB, of 4 MB with page-locked memory, and of a tuned size
@pytest.mark.parametrize("log_m,log_n,shift,block", [(3, 10, 1, 0), (6, 15, 3, 0), (4, 17, 5, 0),
                                                     (5, 14, 7, 1 << 17)])
def test_commit_blocks_any_alignment(lgs, log_m, log_n, shift, block):
    torch = pytest.importorskip("torch")
    ctx = L.Context(0)
    a = rng.field_elements(3, 32 * (64 << log_m)).reshape(32, 64 << log_m)
    pk, _ = L.Ligesis.setup_with_hash(log_m, log_n, L.SubsetSumHash(64 << log_m, a=a), ctx)
    v = rng.field_elements(80 + log_n, 1 << (log_m + log_n))
    dev = torch.from_numpy(v.view(np.int64)).cuda()
    want = L.Ligesis.commit_device(pk, dev.data_ptr(), v.size)[0].root
    ctx.tune(upload_block_bytes=block)
    assert L.Ligesis.commit(pk, L.MlPoly(_unaligned(v, shift)))[0].root == want
    pin = torch.empty(v.size, dtype=torch.int64, pin_memory=True).numpy().view(np.uint64)
    pin[:] = v
    assert L.Ligesis.commit(pk, L.MlPoly(pin))[0].root == want

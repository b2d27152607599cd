"""Commitments of device polynomials whose words are not reduced mod p.  commit_device hands the
caller's words to the row transform as they are (lgs_dft reduces its inputs on the host first), so
these are the transform's own tests at the ends of the 24-bit limbs and beyond p: the codeword
against the oracle's DFT of the reduced values for every row length, and root and proof against
those of the reduced polynomial.  Exact."""
import numpy as np
import pytest

import ligesis_b200 as L
from ligesis_b200 import rng
from tests.helpers import P

pytestmark = pytest.mark.gpu

EDGE = np.array([(1 << 64) - 1, 0, (1 << 24) - 1, ((1 << 24) - 1) << 24, 0xFFFF << 48, P, P - 1,
                 P + 1, 1 << 63, (1 << 48) - 1, P + (1 << 24)], dtype=np.uint64)


def _words(seed, m, n):
    """Rows of 2^64 - 1, of the edges in turn, and of edges at random among any words."""
    w = rng.ints(seed, m * n).reshape(m, n)
    pick = rng.ints(seed + 1, m * n).reshape(m, n)
    w = np.where(pick % np.uint64(3) == 0, w, EDGE[(pick % np.uint64(EDGE.size)).astype(np.int64)])
    w[0] = EDGE[0]
    if m > 1:
        w[1] = EDGE[np.arange(n) % EDGE.size]
    return w


def _reduced(w):
    return np.where(w >= np.uint64(P), w - np.uint64(P), w)


def _commit(pk, w, lend):
    torch = pytest.importorskip("torch")
    dev = torch.from_numpy(w.reshape(-1).view(np.int64)).cuda()
    commit, data = L.Ligesis.commit_device(pk, dev.data_ptr(), w.size, lend=lend)
    return commit.root, data, dev


# 2n = 2^8 (one CTA's shared memory), 2^12 and 2^13 (whole rows), then every final pass, and 2^21
# (the Stockham kernels)
@pytest.mark.parametrize("log_m,log_n", [(2, 7), (2, 11), (2, 12), (2, 13), (2, 14), (2, 15),
                                         (2, 16), (2, 17), (2, 18), (2, 19), (1, 20), (6, 13)])
def test_codeword_of_raw_words(lgs, orc, log_m, log_n):
    m, n = 1 << log_m, 1 << log_n
    hash_ = L.SubsetSumHash(64 * m, a=rng.field_elements(3, 32 * 64 * m).reshape(32, 64 * m))
    pk = L.Ligesis.setup_commit_only(log_m, log_n, hash_, L.Context.default(0))
    w = _words(90 + log_n, m, n)
    root, data, dev = _commit(pk, w, lend=True)
    got = data.codeword()
    for r in sorted({0, 1, m - 1}):
        assert np.array_equal(got[r], orc.dft_bf(_reduced(w[r]), 2 * n)), r
    assert root == _commit(pk, _reduced(w), lend=False)[0]


@pytest.mark.parametrize("log_m,log_n", [(3, 10), (5, 13)])
def test_proof_of_raw_words(lgs, log_m, log_n):
    m = 1 << log_m
    hash_ = L.SubsetSumHash(64 * m, a=rng.field_elements(4, 32 * 64 * m).reshape(32, 64 * m))
    pk, _ = L.Ligesis.setup_with_hash(log_m, log_n, hash_, L.Context.default(0))
    w, z = _words(80, m, 1 << log_n), rng.ext_elements(5, log_m + log_n)
    out = []
    for words in (w, _reduced(w)):
        root, data, dev = _commit(pk, words, lend=True)
        oracle = L.RandomOracle(rng.SeededRng(6), length=2048)
        out.append((root, L.Ligesis.prove(pk, data, z, oracle).data))
    assert out[0] == out[1]

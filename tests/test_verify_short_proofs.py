"""Proofs whose sumchecks have fewer rounds than their vectors have variables, crafted so that every
check before the missing challenges passes: the library's verifier refuses them.  It runs in a child
process, so that a read past the challenges would fail the test and nothing else.  On the CPU."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from ligesis_b200 import proof as codec
from tests.helpers import ligesis_inputs

ROOT = Path(__file__).resolve().parents[1]
ONE = (1, 0)

CHILD = r"""
import ctypes as C, sys
import numpy as np
from ligesis_b200._lib import check, load, ptr64, ptr8
d = np.load(sys.argv[1])
b = lambda k: np.ascontiguousarray(d[k])
com, root, z, proof, fields, ints = (b(k) for k in ("com", "root", "z", "proof", "fields", "ints"))
acc, cur = C.c_int(-1), np.zeros(2, np.uint64)
check(load().lgs_verify(int(d["log_m"]), int(d["log_n"]), ptr8(com), ptr8(root), ptr64(z), len(z),
                        ptr8(proof), proof.size, ptr64(fields), len(fields), ptr64(ints), len(ints),
                        ptr64(cur), C.byref(acc)))
print("accept", acc.value)
"""


@pytest.fixture(scope="module")
def valid(orc):
    log_m, log_n = 3, 10
    f, A, z, fields, ints = ligesis_inputs(log_m, log_n, seed=31)
    key = orc.Key(log_m, log_n, A)
    cm = orc.Commitment(key, f)
    proof, _ = orc.prove(key, cm, z, fields, ints)
    u8 = lambda x: np.frombuffer(x, np.uint8)  # noqa: E731
    return dict(log_m=log_m, log_n=log_n, com=u8(key.com_a), root=u8(cm.root), z=z, fields=fields,
                ints=ints), proof


def _verify(tmp_path, args, proof):
    np.savez(tmp_path / "v.npz", proof=np.frombuffer(proof, np.uint8), **args)
    r = subprocess.run([sys.executable, "-c", CHILD, str(tmp_path / "v.npz")], cwd=ROOT,
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])
    return r.stdout.split()


def test_the_proof_itself_is_accepted(lgs, valid, tmp_path):
    assert _verify(tmp_path, *valid) == ["accept", "1"]


@pytest.mark.parametrize("which", ["sc_recon", "sc_table"])
def test_no_rounds(lgs, valid, tmp_path, which):
    args, proof = valid
    pf = codec.decode(proof)
    sc = pf.sumchecks[which]
    sc.round_polys.clear()  # the claim y4 is then the product of the finals
    if which == "sc_recon":
        sc.final_evals[:] = [pf.y4, ONE]
    else:  # sel over no variables is 1, the other final is y5, and rslink opens that claim
        sc.final_evals[:] = [ONE, pf.y4]
        pf.y5 = pf.y4
        link = pf.sumchecks["sc_rslink"]
        link.round_polys.clear()
        link.final_evals[:] = [pf.y4, ONE]
    assert _verify(tmp_path, args, codec.encode(pf)) == ["accept", "0"]

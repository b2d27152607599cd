"""The engine tuner's choice rests on the engine's own clock: a stand-in engine whose fastest setting
is the one after which the host lingers.  On the CPU."""
import time
from types import SimpleNamespace

import numpy as np

import ligesis_b200 as L
from ligesis_b200 import autotune, engine

BATCH_MS = {(0, 0): 30.0, (0, 74): 20.0, (32, 0): 25.0, (32, 74): 28.0}


class StandIn:
    def __init__(self, device, lanes, tuned):
        assert not tuned

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        return False

    def tune(self, hash_ctas, sumcheck_blocks):
        self.setting = (hash_ctas, sumcheck_blocks)

    def prepare(self, keys):
        assert len(list(keys)) > 0

    def run(self, jobs):
        ms = BATCH_MS[self.setting]
        if self.setting == (0, 74):
            time.sleep(0.05)  # the copies after the last job are no part of the batch
        return [SimpleNamespace(commit=SimpleNamespace(root=bytes([i])),
                                proof=SimpleNamespace(data=bytes([i, 1])),
                                submit_ms=7.0 + 0.1 * i, done_ms=7.0 + ms * (i + 1) / len(jobs))
                for i in range(len(jobs))]


def test_choice_by_the_engines_clock(monkeypatch):
    monkeypatch.setattr(engine, "ProverEngine", StandIn)
    monkeypatch.setattr(L, "Context", lambda device: None)
    monkeypatch.setattr(L, "SubsetSumHash", lambda width, a: None)
    monkeypatch.setattr(L.Ligesis, "setup_with_hash", lambda *a: (object(), None))
    e = autotune.tune_engine(jobs=6, repeats=2, hash_ctas=(0, 32), sumcheck_blocks=(0, 74),
                             save=False)
    assert (e["hash_ctas"], e["sumcheck_blocks"]) == (0, 74)
    got = {(t["hash_ctas"], t["sumcheck_blocks"]): t["pps"] for t in e["trials"]}
    want = {s: 6e3 / ms for s, ms in BATCH_MS.items()}
    assert got.keys() == want.keys()
    assert np.allclose([got[s] for s in want], list(want.values()), atol=0.1)

"""Autotuner for the launch choices of the commit + prove step (lgs_tune), with a JSON cache.

The step runs the commit's subset-sum hash (a persistent tensor-core kernel, one CTA per SM by
default) beside the prove's DAG of sumcheck, eq-table and Basefold kernels, so these choices
trade against each other:

* ``hash_ctas``: how many SMs the hash occupies; fewer leave SMs to the prove's latency-bound
  branches while the hash runs.
* ``sumcheck_blocks``: the grid cap of the multi-CTA sumcheck passes.
* ``hash_groups``: for a polynomial uploaded from host memory, in how many row groups the digest
  is built as the groups' RS encodings finish (under the rest of the upload).

``tune`` times candidate settings on the device (CUDA events on the context's stream): the first
two with f already in HBM (the step the bench's ``value`` times), ``hash_groups`` with f in
page-locked host memory (the step ``e2e`` times).  It keeps the fastest and records it per GPU
name and shape in the cache (``tuning.json`` beside this file unless a path is given).
``apply`` sets a context from the cache.  Every setting computes the same commitment and proof
bytes; ``tune`` checks that too.
"""
from __future__ import annotations

import json
import time
from pathlib import Path

import numpy as np

CACHE = Path(__file__).with_name("tuning.json")
PARAMS = ("hash_ctas", "sumcheck_blocks", "hash_groups")


def _device_name(device: int = 0) -> str:
    import torch

    return torch.cuda.get_device_name(device)


def shape_key(log_m: int, log_n: int) -> str:
    return f"{log_m}x{log_n}"


def load(path: Path | None = None) -> dict:
    p = Path(path or CACHE)
    return json.loads(p.read_text()) if p.exists() else {}


def lookup(log_m: int, log_n: int, device: int = 0, path: Path | None = None) -> dict | None:
    entry = load(path).get(_device_name(device), {}).get(shape_key(log_m, log_n))
    return {k: entry[k] for k in PARAMS if k in entry} if entry else None


def engine_key(lanes: int) -> str:
    return f"engine{lanes}"


def lookup_engine(lanes: int, device: int = 0, path: Path | None = None) -> dict | None:
    entry = load(path).get(_device_name(device), {}).get(engine_key(lanes))
    return {k: entry[k] for k in ("hash_ctas", "sumcheck_blocks") if k in entry} if entry else None


def apply(ctx, log_m: int, log_n: int, path: Path | None = None) -> dict | None:
    """Sets ctx's launch choices from the cache; returns them (None: no entry, defaults kept)."""
    best = lookup(log_m, log_n, ctx.device, path)
    if best:
        ctx.tune(**best)
    return best


def tune(log_m: int, log_n: int, steps: int = 10, warmup: int = 3, repeats: int = 3,
         device: int = 0,
         hash_ctas=None, sumcheck_blocks=None, hash_groups=None, path: Path | None = None,
         save: bool = True) -> dict:
    """Coordinate search: hash_ctas first (sumcheck_blocks at its default), then
    sumcheck_blocks at the best hash_ctas, then hash_groups on the host-input step.  Returns the
    cache entry it wrote."""
    import torch

    import ligesis_b200 as L
    from ligesis_b200 import rng

    torch.cuda.set_device(device)
    sms = torch.cuda.get_device_properties(device).multi_processor_count
    hash_ctas = list(hash_ctas or [sms - d for d in (0, 8, 16, 24, 32, 40, 48, 56)])
    sumcheck_blocks = list(sumcheck_blocks or [296, 222, 148, 74])
    hash_groups = list(hash_groups or [1, 2, 4, 8])
    ctx = L.Context(device)
    stream = torch.cuda.ExternalStream(ctx.stream_ptr, device=torch.device("cuda", device))
    mu = log_m + log_n
    f = rng.field_elements(1, 1 << mu)
    A = rng.field_elements(2, 32 * (64 << log_m)).reshape(32, 64 << log_m)
    z = rng.ext_elements(3, mu)
    g = rng.SeededRng(4)
    oracle = L.RandomOracle(0, length=8)
    oracle.fields, oracle.ints = g.ext_elements(4096), g.ints(4096)
    pk, _ = L.Ligesis.setup_with_hash(log_m, log_n, L.SubsetSumHash(64 << log_m, a=A), ctx)
    f_dev = torch.from_numpy(f.view(np.int64)).to(f"cuda:{device}")
    f_pin = torch.from_numpy(f.view(np.int64)).pin_memory().numpy().view(np.uint64)
    host_input = False

    def step():
        oracle.restart()
        if host_input:
            commit, data = L.Ligesis.commit(pk, L.MlPoly(f_pin))
        else:
            commit, data = L.Ligesis.commit_device(pk, f_dev.data_ptr(), f.size, lend=True)
        proof = L.Ligesis.prove(pk, data, z, oracle)
        return commit, proof

    ref = None

    def measure(setting: dict) -> float:
        nonlocal ref
        ctx.tune(**setting)
        prev = None
        for _ in range(warmup):
            prev = step()
        c, p = prev
        out = (c.root, p.data)
        if ref is None:
            ref = out
        if out != ref:
            raise RuntimeError(f"setting {setting} changed the commitment or proof")
        del prev, c, p
        best_ms = None
        for _ in range(repeats):  # the fastest of `repeats` runs: timing noise only adds
            torch.cuda.synchronize(device)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            for _ in range(steps):
                last = step()
            e1.record(stream)
            torch.cuda.synchronize(device)
            del last
            ms = e0.elapsed_time(e1) / steps
            best_ms = ms if best_ms is None else min(best_ms, ms)
        return best_ms

    trials = []
    best = {"hash_ctas": 0, "sumcheck_blocks": 0}
    best_ms = measure(best)
    trials.append({**best, "ms": round(best_ms, 4)})
    for h in hash_ctas:
        s = {"hash_ctas": h, "sumcheck_blocks": 0}
        ms = measure(s)
        trials.append({**s, "ms": round(ms, 4)})
        if ms < best_ms:
            best, best_ms = s, ms
    for b in sumcheck_blocks:
        s = {"hash_ctas": best["hash_ctas"], "sumcheck_blocks": b}
        ms = measure(s)
        trials.append({**s, "ms": round(ms, 4)})
        if ms < best_ms:
            best, best_ms = s, ms
    host_input = True
    best_e2e, e2e_trials = None, []
    for gcount in hash_groups:
        s = {**best, "hash_groups": gcount}
        ms = measure(s)
        e2e_trials.append({**s, "ms": round(ms, 4)})
        if best_e2e is None or ms < best_e2e[1]:
            best_e2e = (gcount, ms)
    best["hash_groups"] = best_e2e[0]
    ctx.tune(hash_ctas=0, sumcheck_blocks=0, hash_groups=0)
    entry = {**best, "ms": round(best_ms, 4), "default_ms": trials[0]["ms"],
             "e2e_ms": round(best_e2e[1], 4), "e2e_one_group_ms": e2e_trials[0]["ms"],
             "steps": steps, "when": time.strftime("%Y-%m-%d"), "trials": trials,
             "e2e_trials": e2e_trials}
    if save:
        cache = load(path)
        cache.setdefault(_device_name(device), {})[shape_key(log_m, log_n)] = entry
        Path(path or CACHE).write_text(json.dumps(cache, indent=1) + "\n")
    return entry


def tune_engine(lanes: int = 12, jobs: int = 96, repeats: int = 3, device: int = 0,
                hash_ctas=(0, 32, 64), sumcheck_blocks=(0, 37, 74, 148),
                path: Path | None = None, save: bool = True) -> dict:
    """Grid search of the engine lanes' launch choices on the batch workload (`jobs` polynomials
    of mu = floor(14 + 8u), host f in, proof out): with many small jobs in flight, smaller
    hash and sumcheck grids let kernels of different lanes share the SMs.  Keeps the setting
    with the most proofs per second and records it per GPU name under "engine<lanes>"; every
    setting must give the same roots and proofs.  A batch's time is the engine's own, first
    submission to last completion, the best of `repeats`: the copies of the proofs into Python
    afterwards (30 MB a batch) take a third as long again when they land on fresh pages, and
    whether they do depends on what the process holds, not on the setting."""
    import gc

    import ligesis_b200 as L
    from ligesis_b200 import rng
    from ligesis_b200.engine import ProverEngine
    from ligesis_b200.workloads import batch_mus, shape_for_mu

    mus = batch_mus(jobs)
    ctx = L.Context(device)
    keys = {}
    for mu in sorted(set(mus)):
        lm, ln = shape_for_mu(mu)
        A = rng.field_elements(100 + lm, 32 * (64 << lm)).reshape(32, 64 << lm)
        keys[mu] = L.Ligesis.setup_with_hash(lm, ln, L.SubsetSumHash(64 << lm, a=A), ctx)[0]
    work = [(keys[mu], rng.field_elements(1000 + i, 1 << mu), rng.ext_elements(2000 + i, mu))
            for i, mu in enumerate(mus)]
    oracles = [L.RandomOracle(3000 + i, length=1024) for i in range(len(work))]
    trials, ref, best = [], None, None
    with ProverEngine(device, lanes=lanes, tuned=False) as eng:
        for h in hash_ctas:
            for b in sumcheck_blocks:
                eng.tune(hash_ctas=h, sumcheck_blocks=b)
                eng.prepare(keys.values())

                def batch():
                    for o in oracles:
                        o.restart()
                    return eng.run([(pk, f, z, o) for (pk, f, z), o in zip(work, oracles)])

                out = [(r.commit.root, r.proof.data) for r in batch()]  # warm-up
                if ref is None:
                    ref = out
                if out != ref:
                    raise RuntimeError(f"engine setting {h}, {b} changed a root or proof")
                t_best = None
                for _ in range(repeats):
                    gc.collect()
                    gc.disable()
                    res = batch()
                    gc.enable()
                    t = (max(r.done_ms for r in res) - min(r.submit_ms for r in res)) / 1e3
                    t_best = t if t_best is None else min(t_best, t)
                pps = round(len(work) / t_best, 1)
                trials.append({"hash_ctas": h, "sumcheck_blocks": b, "pps": pps})
                if best is None or pps > best["pps"]:
                    best = trials[-1]
    entry = {**best, "default_pps": trials[0]["pps"], "jobs": jobs, "lanes": lanes,
             "when": time.strftime("%Y-%m-%d"), "trials": trials}
    if save:
        cache = load(path)
        cache.setdefault(_device_name(device), {})[engine_key(lanes)] = entry
        Path(path or CACHE).write_text(json.dumps(cache, indent=1) + "\n")
    return entry

"""The prover's work as its users call it, in cases of plain sizes for timing.

A case names one kind of call and its sizes:

  open      `Ligesis.commit` (or `commit_device`) of a 2^log_m x 2^log_n polynomial and
            `Ligesis.prove` at one point: root and proof bytes
  verify    `Ligesis.verify` of such a proof
  commit    `Ligesis.commit_device` under a commit-only key: the root
  batch     jobs of mixed sizes through `ProverEngine.run`: every root and proof
  basefold  `Basefold.commit_{base,ext}_on_domain` and `Basefold.prove`
  lookup    `Lookup.prove_with_opening_points` (GKR-LogUp)
  sumcheck  `lgs_sumcheck_prove_dev` of d multilinear factors over F_{p^2}
  linear    `proofsys.linear_witness` on device tensors
  block     `proofsys.block_witness`, one GPT-2 block from host arrays

`listed()` is the fixed set, `draw` gives more of the same ranges.  `prepare` makes a case's
inputs from its seed, `run` is one pass, `work` what a pass cannot do without.  All results are
whole numbers (exact residues mod p, int64 witnesses, hashes).
"""
from __future__ import annotations

import ctypes

import numpy as np
import torch

import ligesis_b200 as L
from ligesis_b200 import proofsys, rng, workloads
from ligesis_b200._lib import check
from ligesis_b200.engine import ProverEngine

LANES = 12  # the engine's lanes in batch and served proving
PROOF_BYTES = 1 << 20  # room for one proof: its Merkle openings' lengths follow the queries


def listed():
    return [
        # the smallest opening: a served request's latency, launches and host planning
        {"name": "open_3x11", "kind": "open", "log_m": 3, "log_n": 11, "host": True},
        # an ordinary opening of a polynomial the caller holds in host memory (2^20 values)
        {"name": "open_6x14", "kind": "open", "log_m": 6, "log_n": 14, "host": True},
        # the headline: 2^24 values resident in HBM
        {"name": "open_7x17", "kind": "open", "log_m": 7, "log_n": 17, "host": False},
        # the largest opening: 2^26 values
        {"name": "open_7x19", "kind": "open", "log_m": 7, "log_n": 19, "host": False},
        # the other direction: checking a proof of 2^20 values
        {"name": "verify_6x14", "kind": "verify", "log_m": 6, "log_n": 14},
        # square matrices can be committed but not opened: long columns, few of them
        {"name": "commit_12x12", "kind": "commit", "log_m": 12, "log_n": 12},
        # batched proving: independent polynomials of 2^14 .. 2^21 values through the lanes
        {"name": "batch_48", "kind": "batch", "jobs": 48, "mix": 5},
        # the secondary PCS on its own, host polynomial in, proof out
        {"name": "basefold_22", "kind": "basefold", "mu": 22, "ext": False, "rate": 1},
        # the lookup argument of the witness' tables: 2^22 queries into 2^16 entries
        {"name": "lookup_22_16", "kind": "lookup", "mu": 22, "nu": 16, "host": False},
        # the product sumcheck by itself (three factors, as its benchmark runs it)
        {"name": "sumcheck_22_d3", "kind": "sumcheck", "mu": 22, "d": 3},
        # the witness' vocabulary head, transposed weights, ragged in every dimension
        {"name": "linear_head", "kind": "linear", "rows": 31, "inner": 768, "cols": 50257,
         "transposed": True, "bias": False},
        # one transformer block of the integer GPT-2: its four layers, norms, softmax and tables
        {"name": "block_gpt2", "kind": "block", "n_seq": 31, "d_model": 768, "n_head": 12,
         "mlp_hidden": 3072},
    ]


def draw(r):
    kind = r.choice(["open", "open", "verify", "commit", "batch", "basefold", "lookup",
                     "sumcheck", "linear", "linear", "block"])
    if kind in ("open", "verify"):  # inside setup's window log_m + 7 <= log_n <= log_m + 17
        log_m = r.randint(3, 7)
        log_n = r.randint(log_m + 7, min(log_m + 13, 19 if kind == "open" else 17))
        case = {"kind": kind, "log_m": log_m, "log_n": log_n}
        if kind == "open":
            case["host"] = log_m + log_n <= 22 and r.random() < 0.6
        return case
    if kind == "commit":
        log_m = r.randint(4, 12)
        return {"kind": kind, "log_m": log_m, "log_n": r.randint(7, 24 - log_m)}
    if kind == "batch":
        return {"kind": kind, "jobs": r.randint(8, 40), "mix": r.randint(1, 1 << 20)}
    if kind == "basefold":
        ext = r.random() < 0.4
        return {"kind": kind, "mu": r.randint(10, 20 if ext else 22), "ext": ext,
                "rate": r.choice([1, 1, 2, 3])}
    if kind == "lookup":
        mu = r.randint(4, 22)
        return {"kind": kind, "mu": mu, "nu": r.randint(2, min(mu, 16)),
                "host": mu <= 18 and r.random() < 0.5}
    if kind == "sumcheck":
        return {"kind": kind, "mu": r.randint(8, 22), "d": r.randint(1, 3)}
    if kind == "linear":  # log-uniform, odd sizes among them
        return {"kind": kind, "rows": int(2 ** r.uniform(0, 7)), "inner": int(2 ** r.uniform(5, 12)),
                "cols": int(2 ** r.uniform(5, 13)), "transposed": r.random() < 0.5,
                "bias": r.random() < 0.7}
    heads = r.choice([6, 12])
    return {"kind": kind, "n_seq": r.randint(3, 31), "d_model": 64 * heads, "n_head": heads,
            "mlp_hidden": r.choice([1536, 2048, 3072])}


# ---- inputs ------------------------------------------------------------------------------------
def _field(count, seed):
    """`count` uniform Goldilocks values on the GPU, as int64 bit patterns."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    hi = torch.randint(0, 0xFFFFFFFF, (count,), dtype=torch.int64, device="cuda", generator=g)
    lo = torch.randint(0, 1 << 32, (count,), dtype=torch.int64, device="cuda", generator=g)
    return (hi << 32) | lo  # hi < 2^32 - 1, so every value is below p


def _host(t):
    return t.cpu().numpy().view(np.uint64)


def _key(ctx, log_m, log_n, seed, commit_only=False):
    width = L.ligesis.ETA << log_m
    a = _host(_field(L.ligesis.C_ROWS * width, seed))
    hash_ = L.SubsetSumHash(width, a=a.reshape(L.ligesis.C_ROWS, width))
    if commit_only:
        return L.Ligesis.setup_commit_only(log_m, log_n, hash_, ctx)
    return L.Ligesis.setup_with_hash(log_m, log_n, hash_, ctx)


def _oracle(seed, length=2048, queries=None):
    o = L.RandomOracle(rng.SeededRng(seed), length=length)
    if queries is not None:
        o.ints = np.ascontiguousarray(rng.ints(queries, length))
    return o


_engines: dict[int, ProverEngine] = {}


def _engine(lanes):
    """The process' engine, as a server keeps one."""
    if lanes not in _engines:
        _engines[lanes] = ProverEngine(0, lanes=lanes)
    return _engines[lanes]


def _block_cfg(case):
    return dict(proofsys.GPT2_31, n_seq=case["n_seq"], d_model=case["d_model"],
                n_head=case["n_head"], mlp_hidden=case["mlp_hidden"])


def prepare(case, seed):
    kind, ctx = case["kind"], L.Context.default(0)
    s = {"kind": kind, "ctx": ctx, "case": case}
    if kind in ("open", "verify", "commit"):
        log_m, log_n = case["log_m"], case["log_n"]
        f = _field(1 << (log_m + log_n), 7 * seed + 1)
        if kind == "commit":
            s.update(f=f, pk=_key(ctx, log_m, log_n, 7 * seed + 2, commit_only=True))
            return s
        pk, vk = _key(ctx, log_m, log_n, 7 * seed + 2)
        s.update(pk=pk, vk=vk, z=rng.ext_elements(7 * seed + 3, log_m + log_n),
                 oracle=_oracle(7 * seed + 4))
        if kind == "open":
            s["f"] = L.MlPoly(_host(f)) if case["host"] else f
            s["proof"] = np.zeros(PROOF_BYTES, dtype=np.uint8)
            return s
        s["commit"], data = L.Ligesis.commit_device(pk, f.data_ptr(), f.numel())
        s["proof"] = L.Ligesis.prove(pk, data, s["z"], s["oracle"])
        s["y"] = np.array(s["proof"].y, dtype=np.uint64)
        return s
    if kind == "batch":
        s["engine"], mus = _engine(LANES), workloads.batch_mus(case["jobs"], case["mix"])
        shapes = {mu: workloads.shape_for_mu(mu) for mu in sorted(set(mus))}
        keys = {mu: _key(ctx, lm, ln, 7 * seed + lm)[0] for mu, (lm, ln) in shapes.items()}
        s["engine"].prepare(keys.values())
        # each job's query positions come from its place in the batch, so that a job's proof has
        # one length whatever the seed
        s["jobs"] = [(keys[mu], _host(_field(1 << mu, 1000 * seed + i)),
                      rng.ext_elements(1000 * seed + i, mu),
                      _oracle(1000 * seed + 500 + i, 1024, queries=i)) for i, mu in enumerate(mus)]
        return s
    if kind == "basefold":
        n = 1 << case["mu"]
        v = _host(_field(2 * n if case["ext"] else n, 7 * seed + 1))
        s.update(poly=L.MlPoly(v.reshape(n, 2) if case["ext"] else v),
                 point=rng.ext_elements(7 * seed + 2, case["mu"]), oracle=_oracle(7 * seed + 3),
                 proof=np.zeros(PROOF_BYTES, dtype=np.uint8))
        return s
    if kind == "lookup":
        n, m = 1 << case["nu"], 1 << case["mu"]
        t = _field(2 * n, 7 * seed + 1).view(n, 2)
        g = torch.Generator(device="cuda")
        g.manual_seed(7 * seed + 2)
        idx = torch.randint(0, n, (m,), device="cuda", generator=g)
        e = torch.zeros_like(t)
        e[:, 0] = torch.bincount(idx, minlength=n)
        a = t[idx].contiguous()
        s["inputs"] = [_host(x) if case["host"] else x for x in (a, t, e)]
        s["oracle"] = _oracle(7 * seed + 3)
        return s
    if kind == "sumcheck":
        mu, d = case["mu"], case["d"]
        s["polys"] = _field(d * 2 << mu, 7 * seed + 1)
        s["challenges"] = _field(2 * mu, 7 * seed + 2)
        s["stream"] = torch.cuda.ExternalStream(ctx.stream_ptr)
        return s
    g = torch.Generator(device="cuda")
    g.manual_seed(7 * seed + 1)
    if kind == "linear":  # activations within max_v * scale, 16-bit weights
        act, rows, inner, cols = 200 << 12, case["rows"], case["inner"], case["cols"]
        ints = lambda b, shape: torch.randint(-b, b, shape, dtype=torch.int64,  # noqa: E731
                                              device="cuda", generator=g)
        s.update(x=ints(act, (rows, inner)), bias=ints(act, (cols,)) if case["bias"] else None,
                 w=ints(1 << 15, (cols, inner) if case["transposed"] else (inner, cols)))
        return s
    s["cfg"] = _block_cfg(case)
    s["args"] = proofsys.synthetic_block(seed, s["cfg"])
    return s


# ---- one pass ----------------------------------------------------------------------------------
def _bytes(b):
    return np.frombuffer(b, dtype=np.uint8)


def _kept(proof, buf):
    """The proof in the caller's buffer, and its length."""
    buf[:len(proof)] = _bytes(proof)
    return {"proof": buf, "length": len(proof)}


def run(s):
    kind, ctx, case = s["kind"], s["ctx"], s["case"]
    if "oracle" in s:
        s["oracle"].restart()
    if kind == "open":
        if case["host"]:
            commit, data = L.Ligesis.commit(s["pk"], s["f"])
        else:
            commit, data = L.Ligesis.commit_device(s["pk"], s["f"].data_ptr(), s["f"].numel(),
                                                   lend=True)
        proof = L.Ligesis.prove(s["pk"], data, s["z"], s["oracle"])
        return {"root": _bytes(commit.root), **_kept(proof.data, s["proof"])}
    if kind == "verify":
        ok = L.Ligesis.verify(s["vk"], s["commit"], s["z"], s["proof"], s["oracle"])
        return {"accepted": ok, "value": s["y"]}
    if kind == "commit":
        commit, _ = L.Ligesis.commit_device(s["pk"], s["f"].data_ptr(), s["f"].numel(), lend=True)
        return _bytes(commit.root)
    if kind == "batch":
        for job in s["jobs"]:
            job[3].restart()
        done = s["engine"].run(s["jobs"])
        return {"roots": _bytes(b"".join(d.commit.root for d in done)),
                "proofs": [_bytes(d.proof.data) for d in done]}
    if kind == "basefold":
        commit = L.Basefold.commit_ext_on_domain if case["ext"] else L.Basefold.commit_base_on_domain
        state, com = commit(s["poly"], case["rate"], L.ligesis.LOG_INTERLEAVE, ctx)
        proof = L.Basefold.prove(state, s["point"], s["oracle"])
        return {"root": _bytes(com.root), **_kept(proof.data, s["proof"])}
    if kind == "lookup":
        proof, zq, zt = L.Lookup.prove_with_opening_points(*s["inputs"], s["oracle"], ctx)
        return {"proof": _bytes(proof.data), "zq": zq, "zt": zt}
    if kind == "sumcheck":
        mu, d = case["mu"], case["d"]
        with torch.cuda.stream(s["stream"]):
            polys = s["polys"].clone()  # the prover folds its factors in place
            rounds = polys.new_empty((mu, d + 1, 2))
            finals = polys.new_empty((d, 2))
            ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
            check(L.load().lgs_sumcheck_prove_dev(ctx.handle, ptr(polys), d, mu,
                                                  ptr(s["challenges"]), ptr(rounds), ptr(finals)))
        return rounds, finals
    if kind == "linear":
        return proofsys.linear_witness(s["x"], s["w"], s["bias"], proofsys.GPT2_31["scale"],
                                       case["transposed"], ctx)
    x, w, exp_lut, gelu_lut = s["args"]
    return proofsys.block_witness(x, w, exp_lut, gelu_lut, s["cfg"], ctx)


# ---- what a pass cannot do without: inputs read once, results written once, and operations ------
def _open_work(log_m, log_n, prove=True):
    m, n = 1 << log_m, 1 << log_n
    hashed = 2.0 * 32 * (64 * m) * (2 * n)  # H = A B: one add (and one bit test) per entry
    encoded = m * 2 * n * (log_n + 1) * 1.5  # half a product and one add per butterfly output
    proved = 10.0 * m * n if prove else 0.0  # a-bar, eq tables and the sumchecks over B_I
    return {"bytes": 8.0 * m * n + 32, "flops": hashed + encoded + proved}


def work(case):
    kind = case["kind"]
    if kind in ("open", "commit"):
        return _open_work(case["log_m"], case["log_n"], kind == "open")
    if kind == "verify":  # a proof of about 20 KB per variable, each byte hashed
        size = 20e3 * (case["log_m"] + case["log_n"])
        return {"bytes": size, "flops": 16 * size}
    if kind == "batch":
        parts = [_open_work(*workloads.shape_for_mu(mu))
                 for mu in workloads.batch_mus(case["jobs"], case["mix"])]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "basefold":
        words = (2 if case["ext"] else 1) << case["mu"]
        coded = words << case["rate"]
        logn = case["mu"] - 6 + case["rate"]
        return {"bytes": 8.0 * words, "flops": 1.5 * coded * logn + 10.0 * words + 12.0 * coded}
    if kind == "lookup":  # per query about 10 extension products (5 operations each) per level
        m, n = 1 << case["mu"], 1 << case["nu"]
        return {"bytes": 16.0 * (m + 2 * n), "flops": 100.0 * (m + n)}
    if kind == "sumcheck":
        d, size = case["d"], 1 << case["mu"]
        return {"bytes": 16.0 * d * size, "flops": 5.0 * size * (d + d * (d - 1))}
    if kind == "linear":
        r, i, c = case["rows"], case["inner"], case["cols"]
        return {"bytes": 8.0 * (r * i + i * c + 4 * r * c), "flops": 2.0 * r * i * c}
    n, d, h, heads = case["n_seq"], case["d_model"], case["mlp_hidden"], case["n_head"]
    weights = 4 * d * d + 2 * d * h
    arrays = 2 * n * (3 * 3 * d + 3 * d + 2 * d + 3 * h + 2 * d + 6 * d) + 5 * heads * n * n
    return {"bytes": 8.0 * (weights + arrays), "flops": 2.0 * n * weights + 4.0 * n * n * d}

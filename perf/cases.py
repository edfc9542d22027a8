"""The workloads this library is measured on, through its public Python API.

Every case is work that a BitZ prover has the library do: commitments over the shapes the reference
uses (flock's PcsParams defaults, BitZ's 16- and 32-lane profiles, the square 2^a x 2^a matrices of
the benchmark), openings, the forest's grand-product GKR and the batched commit.  All results are
field elements, hashes and proof bytes: whole numbers, equal bit for bit between correct versions.
"""
import ctypes
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(_ROOT, "bitz-poc_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(_ROOT, "bitz-poc_gb300"))

import bitz_gb300 as bz  # noqa: E402
from bitz_gb300 import gkr  # noqa: E402

SHA, B3 = bz.HashKind.SHA256, bz.HashKind.BLAKE3


def listed():
    return [
        # PcsParams' own defaults (SHA-256, 32 lanes, rate 1/2) at the smallest size that is worth a
        # call: launches and latency
        dict(name="commit 2^10 sha r1 l5", kind="commit", log_n=10, rate=1, lanes=5, hash=SHA),
        # a small serving request from host memory: commit, then the opened rows and their
        # multi-proof (the smallest size of the serving mix, square, rate 1/4)
        dict(name="request 2^14 b3 r2 l7", kind="request", log_n=14, rate=2, lanes=7, hash=B3,
             queries=64),
        # BinaryPcs' default geometry: 32 lanes, rate 1/2
        dict(name="commit 2^17 b3 r1 l5", kind="commit", log_n=17, rate=1, lanes=5, hash=B3),
        # BitZ's default profile (custom:1:4, 16 lanes, rate 1/2) at 2^27 committed bits
        dict(name="commit 2^20 b3 r1 l4", kind="commit", log_n=20, rate=1, lanes=4, hash=B3),
        # flock's PcsParams defaults at a large size
        dict(name="commit 2^22 sha r1 l5", kind="commit", log_n=22, rate=1, lanes=5, hash=SHA),
        # an odd shape between the two families: rate 1/8, 256 lanes
        dict(name="commit 2^21 b3 r3 l8", kind="commit", log_n=21, rate=3, lanes=8, hash=B3),
        # the square 2^10 x 2^10 commit
        dict(name="commit 2^20 b3 r2 l10", kind="commit", log_n=20, rate=2, lanes=10, hash=B3),
        # the headline: the square 2^12 x 2^12 commit at rate 1/4
        dict(name="commit 2^24 b3 r2 l12", kind="commit", log_n=24, rate=2, lanes=12, hash=B3),
        # many commitments of uneven sizes in one plan
        dict(name="batch 16x 2^14..2^20", kind="batch", count=16, lo=14, hi=20, rate=2, hash=B3),
        # opening a 2^20-word witness at one point: round 0, ring switch, recursive proof
        dict(name="bit_mle 2^20 l10", kind="bit_mle", log_n=20, rate=2, lanes=10, hash=B3),
        # the full recursive proof of the headline commitment
        dict(name="prove 2^24 l12", kind="prove", log_n=24, rate=2, lanes=12, hash=B3),
        # the forest's grand-product GKR over 2^22 leaves
        dict(name="gkr 2^12x2^10", kind="gkr", t=12, s=10),
    ]


def draw(rng):
    u = rng.random()
    if u < 0.6:
        # every lane count from 1 to 2^12, every rate, both hashes; SHA-256 hashes a row serially
        # and is used with narrow rows
        log_n = rng.randint(8, 23)
        rate = rng.choice([1, 1, 2, 3])
        if rate == 3:
            log_n = min(log_n, 22)
        h = rng.choice([SHA, B3, B3])
        lanes = rng.randint(0, min(log_n - 1, 7 if h == SHA else 12))
        return dict(kind="commit", log_n=log_n, rate=rate, lanes=lanes, hash=h)
    if u < 0.7:
        log_n = rng.randint(10, 20)
        return dict(kind="request", log_n=log_n, rate=rng.choice([1, 2]), lanes=log_n // 2,
                    hash=B3, queries=rng.randint(1, 1 << (log_n // 2)))
    if u < 0.78:
        lo = rng.randint(10, 15)
        return dict(kind="batch", count=rng.randint(2, 24), lo=lo, hi=rng.randint(lo, 20), rate=2,
                    hash=B3)
    if u < 0.94:
        log_n = rng.randint(14, 22)
        return dict(kind=rng.choice(["bit_mle", "prove"]), log_n=log_n, rate=rng.choice([1, 2]),
                    lanes=rng.randint(4, (log_n + 1) // 2), hash=B3)
    return dict(kind="gkr", t=rng.randint(6, 13), s=rng.randint(2, 9))


# ---- inputs and outputs -----------------------------------------------------
class _Transcript:
    """The library's host BLAKE3 transcript as the GKR prover's transcript."""

    def __init__(self):
        self.t = bz.Blake3Transcript()
        self.t.absorb(b"gkr")

    def send(self, stage, msg):
        self.t.absorb(bytes([stage]) + b"".join(np.asarray(m, np.uint64).tobytes() for m in msg))

    def challenge(self, stage):
        return self.t.get_field_challenge()


class _Raw:
    """Device memory of the library for torch.as_tensor."""

    def __init__(self, ptr, shape, typestr, owner):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr,
                                         "version": 3, "strides": None}
        self.owner = owner


def _params(c):
    return bz.PcsParams(c["log_n"] + 7, c["rate"], c["lanes"], c["hash"])


def _open_config(c):
    """initial_k folds every lane; then one recursive step over half of the columns' variables.
    The queries are the rate's unique-decoding count."""
    k, log_n = c["lanes"], c["log_n"]
    left = log_n - k                       # variables after the lane folds
    k1 = max(1, left // 2)
    q = {1: 243, 2: 148}[c["rate"]]
    block0, block1 = 1 << (left + c["rate"]), 1 << (left - k1 + 2)
    return bz.LigeritoConfig(initial_k=k, recursive_ks=[k1], log_inv_rates=[c["rate"], 2],
                             queries=[min(q, block0 // 2), min(148, block1 // 2)],
                             grinding_bits=[16, 8], fold_grinding_bits=None,
                             ood_samples=[0, 1], hash_kind=c["hash"])


def _commitment(params, c, pd):
    cw, tree = pd.device_ptrs()
    return {"root": np.frombuffer(c.root, np.uint8),
            "codeword": torch.as_tensor(_Raw(cw, (params.codeword_len_f128(), 2), "<i8", pd),
                                        device="cuda"),
            "tree": torch.as_tensor(_Raw(tree, (2 * params.n_leaves() - 1, 32), "|u1", pd),
                                    device="cuda")}


def _plan_codeword(plan, i):
    """The resident codeword of commitment i of a plan."""
    cw, tree = ctypes.c_void_p(), ctypes.c_void_p()
    if bz.lib().bz_commitment_device_ptrs(plan.L.bz_batch_plan_commitment(plan.h, i),
                                          ctypes.byref(cw), ctypes.byref(tree)):
        raise RuntimeError("no codeword %d" % i)
    return torch.as_tensor(_Raw(cw.value, (plan.params[i].codeword_len_f128(), 2), "<i8", plan),
                           device="cuda")


def _padded(path, queries, leaves):
    """A multi-proof's length depends on the queries drawn: zero rows up to the longest it can be."""
    out = np.zeros((queries * max(leaves.bit_length() - 1, 1), 32), np.uint8)
    out[:len(path)] = path
    return out


def _proof(p, c, cfg):
    left = c["log_n"] - c["lanes"]
    leaves = [1 << (left + c["rate"]), 1 << (left - cfg.recursive_ks[0] + 2)]
    return {"root": np.frombuffer(bytes(p.initial_root), np.uint8),
            "rows": np.asarray(p.initial_proof.opened_rows),
            "path": _padded(p.initial_proof.merkle_proof, cfg.queries[0], leaves[0]),
            "roots": np.asarray(p.recursive_roots),
            "yr": p.final_proof.yr, "final_rows": np.asarray(p.final_proof.opened_rows),
            "final_path": _padded(p.final_proof.merkle_proof, cfg.queries[1], leaves[1]),
            "sumcheck": p.sumcheck_transcript,
            "nonces": p.grinding_nonces, "ood": p.ood_values}


def prepare(case, seed):
    c = dict(case)
    rng = np.random.default_rng([seed, 20])
    s = {"case": c, "ctx": bz.default_context()}
    kind = c["kind"]
    if kind == "gkr":
        rows, cols = 1 << c["t"], 1 << c["s"]
        s["packed"] = rng.integers(0, 2**64, ((cols + 63) // 64, rows), dtype=np.uint64)
        s["images"] = rng.integers(0, 2**64, (rows, 2), dtype=np.uint64)
        s["zeta"] = [rng.integers(0, 2**64, 2, dtype=np.uint64) for _ in range(c["s"])]
        return s
    if kind == "batch":
        # the sizes are part of the case: the same for every seed
        order = np.random.default_rng([c["count"], c["lo"], c["hi"]])
        sizes = [c["hi"]] + [int(x) for x in order.integers(c["lo"], c["hi"] + 1, c["count"] - 1)]
        s["params"] = [bz.PcsParams(n + 7, c["rate"], n // 2, c["hash"]) for n in sizes]
        s["msgs"] = [bz.DeviceArray.chacha(seed * 64 + i, 1 << n) for i, n in enumerate(sizes)]
        s["plan"] = bz.BatchPlan(s["msgs"], s["params"])
        s["codewords"] = [_plan_codeword(s["plan"], i) for i in range(len(sizes))]
        return s
    s["params"] = _params(c)
    if kind == "request":
        s["msg"] = bz.chacha_words(seed, 1 << c["log_n"])
        s["pos"] = np.sort(rng.choice(s["params"].n_positions(), c["queries"], replace=False))
        return s
    s["msg"] = bz.DeviceArray.chacha(seed, 1 << c["log_n"])
    if kind == "commit":
        return s
    s["config"] = _open_config(c)
    if kind == "prove":
        s["basis"] = bz.DeviceArray.chacha(seed + 1000, 1 << c["log_n"])
        s["target"] = rng.integers(0, 2**64, 2, dtype=np.uint64)
        s["root"], s["data"] = bz.commit(s["msg"], s["params"])
    else:
        s["pcs"] = bz.BinaryPcs(c["log_n"], s["config"], 8)
        s["point"] = rng.integers(0, 2**64, (c["log_n"] + 7, 2), dtype=np.uint64)
        s["root"], s["data"] = s["pcs"].commit(s["msg"])
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "commit":
        if "data" in s:
            s["data"].free()
        c, s["data"] = bz.commit(s["msg"], s["params"])
        return _commitment(s["params"], c, s["data"])
    if kind == "request":
        c, pd = bz.commit(s["msg"], s["params"])
        out = {"root": np.frombuffer(c.root, np.uint8), "rows": pd.rows(s["pos"]),
               "path": _padded(pd.multi_proof(s["pos"]), len(s["pos"]), s["params"].n_leaves())}
        pd.free()
        return out
    if kind == "batch":
        s["plan"].launch()
        return {"roots": np.frombuffer(b"".join(s["plan"].roots()), np.uint8),
                "codewords": s["codewords"]}
    if kind == "gkr":
        roots, point, claim = gkr.forest_prove(s["packed"], s["images"], s["case"]["t"],
                                               s["case"]["s"], s["zeta"], _Transcript())
        return {"roots": roots, "point": np.asarray(point), "claim": claim}
    t = bz.Blake3Transcript()
    t.absorb_slice(s["root"].root)
    if kind == "prove":
        return _proof(bz.prove(t, s["data"], s["msg"], s["basis"], s["target"], s["config"]),
                      s["case"], s["config"])
    r0 = s["pcs"].prove_round0(t, s["msg"])
    o = s["pcs"].open_bit_mle(t, s["msg"], s["data"], r0, s["point"])
    return {"y": r0.y, "s_v": o.s_v, "proof": _proof(o.lig, s["case"], s["config"])}


def _commit_bytes(log_n, rate, lanes):
    leaves = 1 << (log_n - lanes + rate)
    return (16 << log_n) + (16 << (log_n + rate)) + 64 * leaves


def work(case):
    """Bytes of a pass: each input read once, each output written once.  Nothing here is a
    floating-point operation."""
    c = case
    kind = c["kind"]
    if kind == "commit":
        n = _commit_bytes(c["log_n"], c["rate"], c["lanes"])
    elif kind == "request":
        n = _commit_bytes(c["log_n"], c["rate"], c["lanes"]) + c["queries"] * (16 << c["lanes"])
    elif kind == "batch":
        order = np.random.default_rng([c["count"], c["lo"], c["hi"]])
        sizes = [c["hi"]] + [int(x) for x in order.integers(c["lo"], c["hi"] + 1, c["count"] - 1)]
        n = sum(_commit_bytes(k, c["rate"], k // 2) for k in sizes)
    elif kind == "gkr":
        n = (((1 << c["s"]) + 63) // 64) * (8 << c["t"]) + (16 << c["t"]) + (16 << c["s"])
    else:
        # the witness, its basis (written and read once where it is made by the call), the rows
        q = {1: 243, 2: 148}[c["rate"]]
        n = (32 << c["log_n"]) + q * (16 << c["lanes"])
        if kind == "bit_mle":
            n += 16 << c["log_n"]
    return {"bytes": float(n), "flops": 0.0}


def exact(case, seed):
    """No output is a rounded number: all are equal bit for bit or wrong."""
    return None

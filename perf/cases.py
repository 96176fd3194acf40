"""The calls whose speed is measured: whole proofs, the served stream, lifted commitments, transforms, trees, the FRI
chain and the proof-of-work search, each through the package's public entry points.

Every value is an M31 or 32-bit word (or the bytes of a proof), so every output is compared word for word.  The sizes
are those of the repository's benchmark and tests: proofs of 2^10 to 2^24 rows, transforms of 2^12 to 2^24 points,
trees of up to 2^22 leaves, the 34-column lifted commitment.
"""
from __future__ import annotations

import hashlib
import random
import struct

import numpy as np
import torch

from vortexstark_b200 import fri, grind, lifted, merkle, ntt, prover, serving
from vortexstark_b200.circle import Coset

P = 0x7FFFFFFF
COMPRESSION = 80 * 14  # 32-bit operations of one Blake2s compression: 80 G steps of 4 xor, 4 rotations, 6 additions
BUTTERFLY = 3          # a product, a sum and a difference in the field


def listed():
    return [
        # the smallest call a user makes of the prover: one proof, host bytes back, latency and launches count
        {"name": "proof_log10", "kind": "proof", "log_n": 10, "blowup": 2, "queries": 80, "cached": False},
        # an ordinary proof with the largest blowup the tests use, through the kept device state
        {"name": "proof_log17_b3", "kind": "proof", "log_n": 17, "blowup": 3, "queries": 80, "cached": True},
        # the benchmark's headline size
        {"name": "proof_log24", "kind": "proof", "log_n": 24, "blowup": 2, "queries": 80, "cached": True},
        # the benchmark's mixed stream of request sizes through the serving engine, all waiting at once
        {"name": "served_mix", "kind": "served", "requests": 40, "largest": 24, "mix": 7},
        # the benchmark's multi-column commitment: 8 x 2^16, 16 x 2^18 and 10 x 2^20 columns, device-resident
        {"name": "lifted_34cols", "kind": "lifted", "logs": "16*8,18*16,20*10", "blowup": 2, "queries": 80, "host": False},
        # a small commitment of uneven columns in one call from host arrays
        {"name": "lifted_small", "kind": "lifted", "logs": "6*3,9*2,12*6", "blowup": 1, "queries": 20, "host": True},
        # the transform alone, coefficients to values, at the size of the headline's trace
        {"name": "ntt_evaluate_24", "kind": "ntt", "log_n": 24, "inverse": False, "cols": 1, "stwo": False},
        # the other direction on a short column, where the launches and the synchronising call count
        {"name": "ntt_interpolate_16", "kind": "ntt", "log_n": 16, "inverse": True, "cols": 1, "stwo": False},
        # the stwo backend's batched transform of equal columns
        {"name": "stwo_ntt_16x20", "kind": "ntt", "log_n": 20, "inverse": False, "cols": 16, "stwo": True},
        # a root of four columns through the reference's launchers: tiles, node levels, the last block
        {"name": "merkle_tiles_22", "kind": "merkle", "log_n": 22, "cols": 4, "how": "tiles"},
        # every FRI layer of a codeword folded and committed
        {"name": "fri_chain_22", "kind": "fri", "log_n": 22},
        # the proof-of-work search of a stwo proof
        {"name": "grind_24", "kind": "grind", "bits": 24, "m31": False},
    ]


def draw(rng: random.Random):
    kind = rng.choice(["proof", "proof", "served", "lifted", "lifted", "ntt", "ntt", "ntt", "merkle", "merkle", "fri", "grind"])
    if kind == "proof":
        blowup = rng.randint(1, 3)
        return {"kind": kind, "log_n": rng.randint(4, 26 - blowup - 1), "blowup": blowup,
                "queries": rng.choice([1, 20, 70, 80]), "cached": rng.random() < 0.5}
    if kind == "served":
        return {"kind": kind, "requests": rng.randint(1, 40), "largest": rng.choice([16, 18, 20, 22]),
                "mix": rng.randrange(1 << 20)}
    if kind == "lifted":
        host = rng.random() < 0.5
        top = rng.randint(4, 15 if host else 19)
        logs = sorted(rng.sample(range(2, top + 1), rng.randint(1, 3)))
        return {"kind": kind, "logs": ",".join("%d*%d" % (k, rng.randint(1, 14)) for k in logs),
                "blowup": rng.randint(1, 2), "queries": rng.choice([5, 20, 80]), "host": host}
    if kind == "ntt":
        log_n = rng.randint(4, 24)
        return {"kind": kind, "log_n": log_n, "inverse": rng.random() < 0.5,
                "cols": rng.choice([1, 1, rng.randint(2, 20)]) if log_n <= 20 else 1, "stwo": rng.random() < 0.5}
    if kind == "merkle":
        return {"kind": kind, "log_n": rng.randint(10, 22), "cols": rng.randint(1, 16),
                "how": rng.choice(["tiles", "tree", "fused"])}
    if kind == "fri":
        return {"kind": kind, "log_n": rng.randint(4, 23)}
    return {"kind": kind, "bits": rng.randint(10, 25), "m31": rng.random() < 0.5}


def _logs(case):
    out = []
    for part in case["logs"].split(","):
        log_n, count = part.split("*")
        out += [int(log_n)] * int(count)
    return out


def _requests(case):
    """log_n of each request, with the weights of the benchmark's stream."""
    rng = random.Random(case["mix"])
    sizes = [(16, 0.40), (18, 0.25), (20, 0.20), (22, 0.10), (24, 0.05)]
    sizes = [s for s in sizes if s[0] <= case["largest"]]
    got = rng.choices([s[0] for s in sizes], [s[1] for s in sizes], k=case["requests"])
    return [case["largest"]] + got[1:]


def _words(seed, n):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, P, (n,), dtype=torch.int32, device="cuda", generator=g)


def _words8(seed):
    rng = random.Random(seed)
    return [rng.getrandbits(32) for _ in range(8)]


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "proof":
        st = {"a": rng.randrange(P), "b": rng.randrange(P)}
        if case["cached"]:
            st["cache"] = prover.ProverCache(case["log_n"], case["blowup"], case["queries"])
    elif kind == "served":
        logs = _requests(case)
        st = {"inputs": [(k, rng.randrange(P), rng.randrange(P)) for k in logs], "server": serving.ProofServer(16 << 30, 24)}
        for k in sorted(set(logs)):
            st["server"].prewarm(k, min(logs.count(k), 2 if k >= 22 else 6))
    elif kind == "lifted":
        logs = _logs(case)
        gen = np.random.RandomState(seed & 0x7FFFFFFF)
        st = {"columns": [gen.randint(0, P, 1 << k).astype(np.uint32) for k in logs]}
        if not case["host"]:
            st["stream"] = torch.cuda.Stream()
            st["committer"] = lifted.LiftedCommitter(logs, case["blowup"], case["queries"])
            st["committer"].upload_async([c.ctypes.data for c in st["columns"]], st["stream"].cuda_stream)
            st["stream"].synchronize()
    elif kind == "ntt":
        st = {"columns": [_words(seed + 1000 * c, 1 << case["log_n"]) for c in range(case["cols"])]}
        if case["stwo"]:
            st["cache"] = ntt.StwoNttCache(case["log_n"])
        else:
            coset = Coset.half_coset(case["log_n"])
            st["cache"] = ntt.InverseTwiddleCache(coset) if case["inverse"] else ntt.ForwardTwiddleCache(coset)
    elif kind == "merkle":
        st = {"columns": [_words(seed + 1000 * c, 1 << case["log_n"]) for c in range(case["cols"])]}
        if case["how"] == "fused":
            st["root"] = merkle.FusedRoot(case["log_n"])
    elif kind == "fri":
        st = {"columns": [_words(seed + 1000 * c, 1 << case["log_n"]) for c in range(4)],
              "chain": fri.FriChain(case["log_n"]), "state": _words8(seed)}
    else:
        st = {"digest": [w % P if case["m31"] else w for w in _words8(seed)]}
    st["case"] = case
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "proof":
        if case["cached"]:
            blob = prover.prove_cached_bytes(state["a"], state["b"], state["cache"])
        else:
            blob = prover.prove_bytes(state["a"], state["b"], case["log_n"], case["blowup"], case["queries"])
        return np.frombuffer(blob, dtype=np.uint8)
    if kind == "served":
        server, proofs = state["server"], {}
        for tag, (log_n, a, b) in enumerate(state["inputs"]):
            server.submit(tag, log_n, a, b)
        while len(proofs) < len(state["inputs"]):
            for done in server.poll(256, wait_ms=50):
                if done.status:
                    raise RuntimeError("request %d: status %d" % (done.tag, done.status))
                proofs[int(done.tag)] = server.result(int(done.tag))
        return np.frombuffer(b"".join(proofs[t] for t in sorted(proofs)), dtype=np.uint8)
    if kind == "lifted":
        if case["host"]:
            return np.frombuffer(lifted.commit_lifted(state["columns"], case["blowup"], case["queries"]), dtype=np.uint8)
        committer, stream = state["committer"], state["stream"]
        committer.commit_async(stream.cuda_stream, graph=True)
        committer.fetch_async(stream.cuda_stream)
        stream.synchronize()
        return np.frombuffer(committer.result_bytes(), dtype=np.uint8)
    if kind == "ntt":
        cols, cache = state["columns"], state["cache"]
        if case["stwo"]:
            if len(cols) == 1:
                (ntt.interpolate_stwo if case["inverse"] else ntt.evaluate_stwo)(cols[0], cache)
            else:
                (ntt.interpolate_stwo_batch if case["inverse"] else ntt.evaluate_stwo_batch)(cols, cache)
        elif len(cols) == 1:
            (ntt.interpolate if case["inverse"] else ntt.evaluate)(cols[0], cache)
        else:
            (ntt.interpolate_batch if case["inverse"] else ntt.evaluate_batch)(cols, cache)
        return cols
    if kind == "merkle":
        if case["how"] == "fused":
            return state["root"].commit(state["columns"])
        if case["how"] == "tree":
            return merkle.MerkleTree.commit(state["columns"], case["log_n"]).layers
        return merkle.MerkleTree.commit_root_only(state["columns"], case["log_n"])
    if kind == "fri":
        state["chain"].commit_async(state["columns"], state["state"])
        roots, alphas, last = state["chain"].result()
        return [np.array(roots, dtype=np.int64), np.array(alphas, dtype=np.int64), np.array(last, dtype=np.int64)]
    return grind.grind_prefixed(state["digest"], case["bits"], case["m31"])


def _proof_work(log_n, blowup, queries):
    """Trace, quotient and FRI trees of 2N compressions each, one inverse and one extended transform; only the proof's bytes cross."""
    log_e = log_n + blowup
    hashes = 6 << log_e
    flies = (log_n << log_n) // 2 + (log_n << log_e) // 2
    return prover.proof_size(log_n, blowup, queries), hashes * COMPRESSION + flies * BUTTERFLY


def work(case):
    kind = case["kind"]
    if kind == "proof":
        nbytes, flops = _proof_work(case["log_n"], case["blowup"], case["queries"])
    elif kind == "served":
        each = [_proof_work(k, 2, 80) for k in _requests(case)]
        nbytes, flops = sum(e[0] for e in each), sum(e[1] for e in each)
    elif kind == "lifted":
        logs = _logs(case)
        top = max(logs) + case["blowup"]
        flies = sum((k << k) // 2 + (k << (k + case["blowup"])) // 2 for k in logs)
        hashes = ((len(logs) + 15) // 16 + 1 << top) + (2 << top) + (2 << top)
        nbytes = sum(4 << k for k in logs) + lifted.lifted_size(logs, case["blowup"], case["queries"])
        flops = hashes * COMPRESSION + flies * BUTTERFLY
    elif kind == "ntt":
        n = 1 << case["log_n"]
        nbytes = 8 * n * case["cols"] + 4 * n  # each column read and written, the twiddles read
        flops = case["cols"] * case["log_n"] * (n // 2) * BUTTERFLY
    elif kind == "merkle":
        n = 1 << case["log_n"]
        nbytes = 4 * n * case["cols"] + (64 * n if case["how"] == "tree" else 32)
        flops = 2 * n * COMPRESSION
    elif kind == "fri":
        n = 1 << case["log_n"]
        nbytes = 16 * n + 4 * n
        flops = 2 * n * COMPRESSION
    else:
        nbytes = 40
        flops = COMPRESSION << case["bits"]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    return "exact"  # whole words: field elements, digests, proof bytes


def _hash(words):
    return struct.unpack("<8I", hashlib.blake2s(struct.pack("<%dI" % len(words), *words)).digest())


def exact(case, seed):
    """Small trees and searches again with hashlib; the larger ones, and the proofs, take the host too long."""
    if case["kind"] == "merkle" and case["log_n"] <= 16 and case["how"] != "tree":
        cols = [_words(seed + 1000 * c, 1 << case["log_n"]).tolist() for c in range(case["cols"])]
        level = [_hash(row) for row in zip(*cols)]
        while len(level) > 1:
            level = [_hash(level[i] + level[i + 1]) for i in range(0, len(level), 2)]
        return level[0]
    if case["kind"] == "grind" and case["bits"] <= 18:
        digest = [w % P if case["m31"] else w for w in _words8(seed)]
        head = struct.pack("<8I", *digest)
        for i in range(1 << 24):
            nonce = ((i >> 20) << 32) | (i & 0xFFFFF)
            h = struct.unpack("<4I", hashlib.blake2s(head + struct.pack("<Q", nonce)).digest()[:16])
            if case["m31"]:
                h = [w % P for w in h]
            if (h[0] | h[1] << 32 | h[2] << 64 | h[3] << 96) % (1 << case["bits"]) == 0:
                return nonce
    return None

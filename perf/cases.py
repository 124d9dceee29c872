"""Performance cases of the commit-and-fold library, through its public plan API.

Each case is one call sequence a prover's program makes: hash and Merkle plans on
device buffers, the Circle FFT and FRI fold plans between them, whole PCS/FRI
proofs from host coefficients to proof bytes, the batched superstep, the
multilinear sum-check and the proof server.  Every output is exact (digests, field
elements, proof bytes).

listed() are fixed sizes of each call; draw(rng) gives further sizes of the same
ranges; prepare(case, seed) makes the inputs and the plan; run(state) is one pass;
work(case) is the traffic and the integer operations a pass cannot do without.
"""
from __future__ import annotations

import hashlib

import numpy as np
import torch

import apple_b200 as az

P = (1 << 31) - 1
OPS_PER_PERMUTATION = 4320  # 24 rounds of 180 32-bit logic and shift operations
OPS_PER_M31_MUL = 4         # wide multiply, fold (2), final reduction
PUBLIC = bytes(range(32))

_context = None


def context():
    """One library context per program, as with any device handle."""
    global _context
    if _context is None:
        _context = az.Context(0)
    return _context


def listed():
    return [
        # Leaf and nullifier hashing: many short records of one odd length, packed
        # on 8-byte boundaries (SHA3-256, device to device).
        {"name": "hash-100003x100", "kind": "hash", "count": 100003, "length": 100, "stride": 104, "keccak": False},
        # The smallest commitments: a 1024-leaf tree of digests, where latency is all.
        {"name": "merkle-2^10x32", "kind": "merkle", "log": 10, "length": 32, "stride": 32},
        # A full trace commitment: 64-byte leaves at the scale of the hash benchmark.
        {"name": "merkle-2^22x64", "kind": "merkle", "log": 22, "length": 64, "stride": 64},
        # Codeword evaluation of extension-field coefficients already on the device.
        {"name": "codeword-2^20", "kind": "codeword", "log": 20},
        # The bare FRI fold chain with the verifier's challenges known (device to device).
        {"name": "fold-chain-2^22", "kind": "fold_chain", "log": 22, "rounds": 16},
        # Commit-and-fold of an evaluated layer with transcript challenges, layers kept
        # for the query phase.
        {"name": "merkle-chain-2^16", "kind": "merkle_chain", "log": 16, "rounds": 10, "queries": 64},
        # A small proof: host coefficients in the extension field to proof bytes.
        {"name": "pcs-2^10", "kind": "pcs", "log": 10, "rounds": 4, "queries": 32, "blowup": 2, "lifted": False},
        # The standard large proof: 2^20 base-field coefficients, blowup 4, 64 queries.
        {"name": "pcs-2^22", "kind": "pcs", "log": 22, "rounds": 16, "queries": 64, "blowup": 2, "lifted": True},
        # The same statement given as the monomial polynomial P(x) + y Q(x).
        {"name": "polynomial-2^22", "kind": "polynomial", "log": 22, "rounds": 16, "queries": 64, "columns": 1 << 19, "lifted": True},
        # One superstep over uneven instances, host coefficients to host proofs.
        {"name": "batch-128x10-20", "kind": "batch", "instances": 128, "low": 10, "high": 20, "mix": 1, "queries": 64},
        # A multilinear sum-check over a mid-size table on the host.
        {"name": "sumcheck-2^18", "kind": "sumcheck", "log": 18},
        # The server under a burst of small proofs with sum-checks in between (4 : 1).
        {"name": "server-40-jobs", "kind": "server", "proofs": 32, "tables": 8, "low": 12, "high": 16, "table_log": 14, "mix": 1, "queries": 64},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(2.0 ** rng.uniform(lo, hi)))


def draw(rng):
    kind = rng.choice(["hash", "merkle", "codeword", "fold_chain", "merkle_chain", "pcs", "pcs", "polynomial", "batch", "sumcheck", "server"])
    if kind == "hash":
        length = rng.randint(1, 136)
        return {"kind": kind, "count": _log_uniform(rng, 4, 22), "length": length, "stride": length + rng.choice([0, -length % 8, 3]),
                "keccak": rng.random() < 0.25}
    if kind == "merkle":
        length = rng.choice([32, 64, rng.randint(1, 136)])
        return {"kind": kind, "log": rng.randint(4, 22), "length": length, "stride": length + rng.choice([0, -length % 8, 5])}
    if kind == "codeword":
        return {"kind": kind, "log": rng.randint(4, 22)}
    if kind in ("fold_chain", "merkle_chain"):
        log = rng.randint(6, 22 if kind == "fold_chain" else 20)
        case = {"kind": kind, "log": log, "rounds": rng.randint(1, log - 4)}
        if kind == "merkle_chain":
            case["queries"] = rng.randint(16, 80)
        return case
    if kind in ("pcs", "polynomial"):
        log = rng.randint(8, 22)
        case = {"kind": kind, "log": log, "rounds": rng.randint(max(1, log - 8), log - 4), "queries": rng.randint(16, 80), "lifted": rng.random() < 0.5}
        if kind == "pcs":
            case["blowup"] = rng.randint(1, 3)
        else:
            case["columns"] = _log_uniform(rng, log - 5, log - 3)
        return case
    if kind == "batch":
        low = rng.randint(8, 14)
        return {"kind": kind, "instances": rng.randint(8, 128), "low": low, "high": low + rng.randint(2, 6), "mix": rng.randrange(1 << 20),
                "queries": rng.randint(16, 64)}
    if kind == "sumcheck":
        return {"kind": kind, "log": rng.randint(4, 20)}
    low = rng.randint(10, 14)
    return {"kind": kind, "proofs": rng.randint(8, 40), "tables": rng.randint(2, 10), "low": low, "high": low + rng.randint(1, 3),
            "table_log": rng.randint(10, 16), "mix": rng.randrange(1 << 20), "queries": rng.randint(16, 64)}


# ---- shapes ----
def _final_log(log):
    return 6 if log > 6 else log - 1


def _batch_logs(case):
    return [int(v) for v in np.random.default_rng(case["mix"]).integers(case["low"], case["high"] + 1, case["instances"])]


def _server_logs(case):
    """Sizes skewed toward small: P(k) proportional to 2^(-(k - low) / 2)."""
    sizes = np.arange(case["low"], case["high"] + 1)
    p = 2.0 ** (-(sizes - case["low"]) / 2)
    return [int(v) for v in np.random.default_rng(case["mix"]).choice(sizes, case["proofs"], p=p / p.sum())]


# ---- inputs ----
def _bytes_on_device(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=g)


def _field_on_device(n, seed):
    """n QM31 values: 4 canonical M31 limbs each."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, P, (n, 4), dtype=torch.int32, device="cuda", generator=g)


def _field_on_host(rng, n, lifted):
    """n QM31 values on the host; lifted: base-field values (b = c = d = 0)."""
    if not lifted:
        return rng.integers(0, P, (n, 4), dtype=np.uint32)
    v = np.zeros((n, 4), np.uint32)
    v[:, 0] = rng.integers(0, P, n, dtype=np.uint32)
    return v


def _byte_array(data):
    return np.frombuffer(data, np.uint8)


def prepare(case, seed):
    ctx, kind = context(), case["kind"]
    s = {"kind": kind}
    if kind == "hash":
        s["plan"] = az.SHA3FixedOneBlockHashPlan(ctx, case["count"], case["stride"], case["length"], keccak=case["keccak"])
        s["in"] = _bytes_on_device(case["count"] * case["stride"], seed)
        s["out"] = torch.empty(case["count"] * 32, dtype=torch.uint8, device="cuda")
    elif kind == "merkle":
        n = 1 << case["log"]
        s["plan"] = az.SHA3RawLeavesMerkleCommitPlan(ctx, n, case["stride"], case["length"])
        s["in"] = _bytes_on_device(n * case["stride"], seed)
    elif kind == "codeword":
        n = 1 << case["log"]
        s["plan"] = az.CircleCodewordPlan(ctx, case["log"])
        s["in"] = _field_on_device(n, seed)
        s["out"] = torch.empty((n, 4), dtype=torch.int32, device="cuda")
    elif kind == "fold_chain":
        n, r = 1 << case["log"], case["rounds"]
        s["plan"] = az.CircleFRIFoldChainPlan(ctx, case["log"], r)
        s["in"] = _field_on_device(n, seed)
        s["challenges"] = np.random.default_rng(seed).integers(0, P, (r, 4), dtype=np.uint32)
        s["out"] = torch.empty((n >> r, 4), dtype=torch.int32, device="cuda")
    elif kind == "merkle_chain":
        n, r = 1 << case["log"], case["rounds"]
        s["plan"] = az.CircleFRIMerkleTranscriptFoldChainPlan(ctx, case["log"], 2, case["queries"], PUBLIC, r)
        s["in"] = _field_on_device(n, seed)
        s["layers"] = torch.empty((s["plan"].total_committed_layer_count, 4), dtype=torch.int32, device="cuda")
        s["roots"] = torch.empty(32 * r, dtype=torch.uint8, device="cuda")
        s["out"] = torch.empty((n >> r, 4), dtype=torch.int32, device="cuda")
    elif kind == "pcs":
        s["plan"] = az.CirclePCSFRIProver(ctx, case["log"], case["blowup"], case["queries"], case["rounds"])
        s["in"] = _field_on_host(np.random.default_rng(seed), (1 << case["log"]) >> case["blowup"], case["lifted"])
    elif kind == "polynomial":
        rng = np.random.default_rng(seed)
        s["plan"] = az.CirclePCSFRIProver(ctx, case["log"], 2, case["queries"], case["rounds"])
        s["x"] = _field_on_host(rng, case["columns"], case["lifted"])
        s["y"] = _field_on_host(rng, case["columns"], case["lifted"])
    elif kind == "batch":
        rng, logs = np.random.default_rng(seed), _batch_logs(case)
        s["plan"] = az.BatchProver(ctx, logs, [lg - _final_log(lg) for lg in logs], 2, case["queries"])
        s["counts"] = [(1 << lg) >> 2 for lg in logs]
        s["offsets"] = list(np.cumsum([0] + s["counts"][:-1]))
        s["in"] = _field_on_host(rng, sum(s["counts"]), True)
        s["public"] = PUBLIC * len(logs)
    elif kind == "sumcheck":
        s["ctx"] = ctx
        s["in"] = np.random.default_rng(seed).integers(0, P, 1 << case["log"], dtype=np.uint32)
    elif kind == "server":
        rng, logs = np.random.default_rng(seed), _server_logs(case)
        s["queries"] = case["queries"]
        s["server"] = az.ProofServer(ctx, 24 << 30, slots=4)
        shapes = sorted({(lg, lg - _final_log(lg)) for lg in logs})
        s["server"].warm(shapes, log_blowup=2, queries=case["queries"], sumcheck_logs=[case["table_log"]])
        proofs = [("pcs", lg, _field_on_host(rng, (1 << lg) >> 2, True)) for lg in logs]
        tables = [("table", case["table_log"], rng.integers(0, P, 1 << case["table_log"], dtype=np.uint32)) for _ in range(case["tables"])]
        # tables spread evenly between the proofs, in arrival order
        every = max(1, len(proofs) // max(1, len(tables)))
        jobs = []
        for i, job in enumerate(proofs):
            jobs.append(job)
            if i % every == every - 1 and tables:
                jobs.append(tables.pop())
        s["jobs"] = jobs + tables
    else:
        raise ValueError(kind)
    return s


def run(s):
    kind = s["kind"]
    if kind == "hash":
        s["plan"].hash_resident(s["in"].data_ptr(), s["out"].data_ptr())
        return s["out"]
    if kind == "merkle":
        return _byte_array(s["plan"].commit_resident(s["in"].data_ptr()))
    if kind == "codeword":
        s["plan"].execute_resident(s["in"].data_ptr(), s["out"].data_ptr())
        return s["out"]
    if kind == "fold_chain":
        s["plan"].execute_resident(s["in"].data_ptr(), s["out"].data_ptr(), s["challenges"])
        return s["out"]
    if kind == "merkle_chain":
        s["plan"].execute_resident(s["in"].data_ptr(), s["roots"].data_ptr(), s["out"].data_ptr(), dev_committed_layers=s["layers"].data_ptr())
        return [s["out"], s["roots"], s["layers"], s["plan"].challenges()]
    if kind == "pcs":
        return _byte_array(s["plan"].prove_coefficients(s["in"], PUBLIC))
    if kind == "polynomial":
        return _byte_array(s["plan"].prove_polynomial(s["x"], s["y"], PUBLIC))
    if kind == "batch":
        s["plan"].upload(s["in"], s["offsets"], s["counts"])
        s["plan"].prove(s["public"])
        return _byte_array(b"".join(s["plan"].proofs()))
    if kind == "sumcheck":
        r = az.sumcheck_prove(s["ctx"], s["in"])
        return [r["r0"], r["r1"], r["challenges"], r["claimed_sum"], r["final"], _byte_array(r["initial_digest"])]
    server, ids = s["server"], []
    for what, lg, words in s["jobs"]:
        if what == "pcs":
            ids.append(server.submit_pcs(lg, 2, s["queries"], lg - _final_log(lg), words, PUBLIC, copy=False))
        else:
            ids.append(server.submit_sumcheck(words, copy=False))
    server.wait_all()
    proofs, tables = [], []
    for (what, _, _), job in zip(s["jobs"], ids):
        result, _ = server.poll(job)
        if what == "pcs":
            proofs.append(result)
        else:
            tables.append(np.concatenate([result["r0"], result["r1"], result["challenges"],
                                          np.array([result["claimed_sum"], result["final"]], np.uint32),
                                          np.frombuffer(result["initial_digest"], np.uint32)]))
    return [_byte_array(b"".join(proofs)), np.concatenate(tables)]


# ---- what a pass cannot do without ----
def _tree_permutations(log):
    return 2 * (1 << log) - 1


def _fft_muls(log, limbs):
    return log * (1 << log) // 2 * limbs


def _proof_work(log, rounds, queries, coefficients, lifted):
    """Bytes and operations of one commit-and-fold proof."""
    n = 1 << log
    perms = sum(_tree_permutations(log - k) + 3 for k in range(rounds))
    muls = _fft_muls(log, 1 if lifted else 4) + 20 * (n - (n >> rounds))
    return 16 * coefficients + az.pcs_proof_size(log, rounds, queries), OPS_PER_PERMUTATION * perms + OPS_PER_M31_MUL * muls


def _sumcheck_work(log):
    n = 1 << log
    return 4 * n, OPS_PER_PERMUTATION * ((50 + 4 * n) // 136 + 1 + 2 * log) + OPS_PER_M31_MUL * 2 * n


def work(case):
    kind = case["kind"]
    if kind == "hash":
        perms = 2 if case["length"] == 136 else 1
        return {"bytes": case["count"] * (case["length"] + 32), "flops": case["count"] * perms * OPS_PER_PERMUTATION}
    if kind == "merkle":
        n = 1 << case["log"]
        leaf = 2 if case["length"] == 136 else 1
        return {"bytes": n * case["length"] + 32, "flops": OPS_PER_PERMUTATION * (n * leaf + n - 1)}
    n = 1 << case.get("log", 0)
    if kind == "codeword":
        return {"bytes": 32 * n, "flops": OPS_PER_M31_MUL * _fft_muls(case["log"], 4)}
    if kind == "fold_chain":
        out = n >> case["rounds"]
        return {"bytes": 16 * (n + out), "flops": OPS_PER_M31_MUL * 20 * (n - out)}
    if kind == "merkle_chain":
        out = n >> case["rounds"]
        perms = sum(_tree_permutations(case["log"] - k) + 3 for k in range(case["rounds"]))
        return {"bytes": 16 * (n + 2 * (n - out) + out), "flops": OPS_PER_PERMUTATION * perms + OPS_PER_M31_MUL * 20 * (n - out)}
    if kind == "pcs":
        b, f = _proof_work(case["log"], case["rounds"], case["queries"], n >> case["blowup"], case["lifted"])
        return {"bytes": b, "flops": f}
    if kind == "polynomial":
        b, f = _proof_work(case["log"], case["rounds"], case["queries"], 2 * case["columns"], case["lifted"])
        return {"bytes": b, "flops": f}
    if kind == "batch":
        each = [_proof_work(lg, lg - _final_log(lg), case["queries"], (1 << lg) >> 2, True) for lg in _batch_logs(case)]
    elif kind == "sumcheck":
        each = [_sumcheck_work(case["log"])]
    else:
        each = [_proof_work(lg, lg - _final_log(lg), case["queries"], (1 << lg) >> 2, True) for lg in _server_logs(case)]
        each += [_sumcheck_work(case["table_log"])] * case["tables"]
    return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}


def exact(case, seed):
    """Digests and roots by hashlib, at sizes it handles in seconds; the field
    outputs and proofs are exact integers by construction and have no other value."""
    if case["kind"] == "hash" and not case["keccak"] and case["count"] <= 1 << 20:
        m = _bytes_on_device(case["count"] * case["stride"], seed).cpu().numpy().reshape(case["count"], -1)[:, : case["length"]]
        return torch.from_numpy(_byte_array(b"".join(hashlib.sha3_256(r.tobytes()).digest() for r in m)).copy())
    if case["kind"] == "merkle" and case["log"] <= 18:
        n = 1 << case["log"]
        m = _bytes_on_device(n * case["stride"], seed).cpu().numpy().reshape(n, -1)[:, : case["length"]]
        level = [hashlib.sha3_256(r.tobytes()).digest() for r in m]
        while len(level) > 1:
            level = [hashlib.sha3_256(level[i] + level[i + 1]).digest() for i in range(0, len(level), 2)]
        return _byte_array(level[0])
    return None

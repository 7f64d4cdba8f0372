"""The work that programs built on this backend have it do, as measurable cases.

Each kind below is one way a program uses the backend, through the entry
points of `gpustark`: whole proofs (`prove`), the proof server (`serve`), a
batched commitment of columns of mixed sizes (`plan`), and the operations of
the backend traits as a generic prover calls them: low-degree extension
(`lde`), a Merkle commitment (`merkle`), many small commitments at once
(`worklist`), a FRI commit phase (`fri`), and out-of-domain evaluation with
the DEEP quotients (`deep`). All values are M31 words (32-bit integers) or
hash bytes, and the arithmetic is exact.
"""
import functools
import hashlib
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nitroozk-stwo_b200"))

from gpustark import prove as G  # noqa: E402
from gpustark import serve as S  # noqa: E402
from gpustark.backend import CommitPlan, GpuBackend as B  # noqa: E402

P = (1 << 31) - 1


def listed():
    return [
        # the smallest proof of the batched workload: latency and launches
        {"name": "prove_wf_2e10x16", "kind": "prove", "air": "wide_fibonacci", "log": 10, "cols": 16, "host": True,
         "channel": "blake2s", "blowup": 1, "queries": 70},
        # the Wide-Fibonacci benchmark proof, its two input columns on the host
        {"name": "prove_wf_2e16x100", "kind": "prove", "air": "wide_fibonacci", "log": 16, "cols": 100, "host": True,
         "channel": "blake2s", "blowup": 1, "queries": 70},
        # the headline benchmark proof, inputs generated on the device
        {"name": "prove_poseidon_2e18", "kind": "prove", "air": "poseidon", "log": 18, "cols": 158, "host": False,
         "channel": "blake2s", "blowup": 1, "queries": 70},
        # the same Wide-Fibonacci proof over the second channel (felt252 hashes for a recursive verifier)
        {"name": "prove_wf_2e16x100_p252", "kind": "prove", "air": "wide_fibonacci", "log": 16, "cols": 100,
         "host": True, "channel": "poseidon252", "blowup": 1, "queries": 70},
        # the batched workload: 64 independent small proofs in flight at once
        {"name": "serve_64_wf", "kind": "serve", "jobs": 64, "lo": 10, "hi": 16},
        # the batched commitment workload: 256 trace columns of log sizes 12..24, one tree
        {"name": "plan_256_12to24", "kind": "plan", "cols": 256, "lo": 12, "hi": 24, "blowup": 1},
        # a proof's dominant transform: the Poseidon2 trace interpolated and extended to the constraint domain
        {"name": "lde_158x2e18_b2", "kind": "lde", "cols": 158, "log": 18, "blowup": 2},
        # one long column, evaluated on its own domain: the transform sweep
        {"name": "lde_1x2e24_b0", "kind": "lde", "cols": 1, "log": 24, "blowup": 0},
        # a Merkle commitment of the kernel sweep's shape
        {"name": "merkle_64x2e20", "kind": "merkle", "cols": 64, "log": 20},
        # commitments of many small components: transforms and trees of uneven sizes in one call each
        {"name": "worklist_32x4to9", "kind": "worklist", "trees": 32, "cols": 8, "lo": 4, "hi": 9},
        # a FRI commit phase driven from the host, one trait call per step
        {"name": "fri_2e22", "kind": "fri", "log": 22},
        # out-of-domain values and DEEP quotients of a Wide-Fibonacci trace
        {"name": "deep_100x2e17", "kind": "deep", "cols": 100, "log": 17},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["prove", "prove", "prove", "lde", "lde", "merkle", "fri", "deep", "plan", "serve", "worklist"])
    if kind == "prove":
        blowup = rng.choice([1, 1, 1, 2])
        if rng.random() < 0.5:
            log = rng.randint(6, 18 if blowup == 1 else 16)
            c = {"air": "poseidon", "log": log, "cols": 158}
        else:
            log = rng.randint(5, 17)
            c = {"air": "wide_fibonacci", "log": log, "cols": _log_uniform(rng, 5, 160)}
        channel = "poseidon252" if c["log"] <= 16 and rng.random() < 0.25 else "blake2s"
        return {"kind": kind, **c, "host": rng.random() < 0.5, "channel": channel, "blowup": blowup,
                "queries": rng.choice([3, 30, 70])}
    if kind == "serve":
        lo = rng.randint(8, 11)
        return {"kind": kind, "jobs": rng.randint(4, 64), "lo": lo, "hi": rng.randint(lo, 15)}
    if kind == "plan":
        lo = rng.randint(4, 12)
        return {"kind": kind, "cols": _log_uniform(rng, 9, 256), "lo": lo, "hi": rng.randint(lo + 4, 22),
                "blowup": rng.choice([1, 1, 2])}
    if kind == "lde":
        log, blowup = rng.randint(4, 24), rng.choice([0, 1, 1, 2])
        most = max(1, min(256, (158 << 20) >> (log + blowup)))
        return {"kind": kind, "cols": _log_uniform(rng, 1, most), "log": log, "blowup": blowup}
    if kind == "merkle":
        log = rng.randint(5, 22)
        return {"kind": kind, "cols": _log_uniform(rng, 1, max(1, min(300, (64 << 20) >> log))), "log": log}
    if kind == "fri":
        return {"kind": kind, "log": rng.randint(5, 22)}
    if kind == "deep":
        log = rng.randint(5, 20)
        return {"kind": kind, "cols": _log_uniform(rng, 2, min(200, (200 << 17) >> log)), "log": log}
    lo = rng.randint(3, 6)
    return {"kind": "worklist", "trees": rng.randint(3, 48), "cols": rng.randint(1, 12), "lo": lo,
            "hi": rng.randint(lo, 9)}


# --------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _columns(g, n_cols, log):
    """n_cols columns of 2^log uniform M31 values, as rows of one tensor."""
    return torch.randint(0, P, (n_cols, 1 << log), dtype=torch.int32, device="cuda", generator=g)


def _host_columns(g, n_cols, log):
    """The same in pinned host memory, as the array the provers take."""
    return _columns(g, n_cols, log).cpu().pin_memory().numpy().view(np.uint32)


@functools.lru_cache(maxsize=None)
def _twiddles(root_log):
    return B.precompute_twiddles(root_log)


@functools.lru_cache(maxsize=None)
def _server():
    return S.ProofServer(4, 96 << 30, fibers_per_worker=6)


def _qm31(rnd):
    return [rnd.randrange(P) for _ in range(4)]


def _plan_logs(case):
    rnd = random.Random(7)
    logs = [rnd.randint(case["lo"], case["hi"]) for _ in range(case["cols"])]
    logs[0] = case["hi"]
    return logs


def _tree_logs(case):
    rnd = random.Random(11)
    return [rnd.randint(case["lo"], case["hi"]) for _ in range(case["trees"])]


def _jobs(case):
    rnd = random.Random(13)
    return [(rnd.randint(case["lo"], case["hi"]), rnd.randint(16, 100)) for _ in range(case["jobs"])]


def _proof_bound(log, cols, blowup, queries):
    """No proof of this shape is longer: per query, a path in every tree, the
    FRI layers' paths and witnesses and every column's value."""
    depth = log + blowup + 2
    return queries * (16 * depth * depth + 112 * depth + 4 * cols + 64) + 20 * cols + 4000


def prepare(case, seed):
    g, rnd, kind = _gen(seed), random.Random(seed), case["kind"]
    s = {"kind": kind}
    if kind == "prove":
        s.update(case=case, seed=seed, config=G.pcs_config(n_queries=case["queries"], log_blowup=case["blowup"]))
        if case["host"]:
            s["inputs"] = _host_columns(g, 16 if case["air"] == "poseidon" else 2, case["log"])
        s.update(out=np.zeros(_proof_bound(case["log"], case["cols"], case["blowup"], case["queries"]), np.uint8), n=0)
    elif kind == "serve":
        s.update(server=_server(), jobs=[(log, cols, rnd.randrange(1 << 32)) for log, cols in _jobs(case)])
        s.update(out=np.zeros(sum(_proof_bound(log, cols, 1, 70) for log, cols in _jobs(case)), np.uint8), n=0)
    elif kind == "plan":
        logs = _plan_logs(case)
        s.update(plan=CommitPlan(logs, case["blowup"]), columns=[_columns(g, 1, log)[0] for log in logs])
    elif kind == "lde":
        log, out_log = case["log"], case["log"] + case["blowup"]
        s.update(log=log, out_log=out_log, tw=_twiddles(out_log - 1), trace=_columns(g, case["cols"], log))
        s["evals"] = torch.empty(case["cols"], 1 << out_log, dtype=torch.int32, device="cuda")
    elif kind == "merkle":
        s.update(log=case["log"], columns=_columns(g, case["cols"], case["log"]))
        s["layers"] = [torch.empty(8 << k, dtype=torch.int32, device="cuda") for k in range(case["log"] + 1)]
    elif kind == "worklist":
        logs = _tree_logs(case)
        s.update(tw=_twiddles(max(logs)), logs=logs, traces=[_columns(g, case["cols"], k) for k in logs])
        s["coeffs"] = [torch.empty_like(t) for t in s["traces"]]
        s["evals"] = [torch.empty(case["cols"], 2 << k, dtype=torch.int32, device="cuda") for k in logs]
    elif kind == "fri":
        s.update(log=case["log"], tw=_twiddles(case["log"] - 1), planes=_columns(g, 4, case["log"]),
                 alpha=_qm31(rnd))
    elif kind == "deep":
        n = case["cols"]
        s.update(log=case["log"], coeffs=_columns(g, n, case["log"]), evals=_columns(g, n, case["log"] + 1),
                 point=_qm31(rnd) + _qm31(rnd), b=[_qm31(rnd) for _ in range(n)], c=[_qm31(rnd) for _ in range(n)],
                 first=_qm31(rnd))
    return s


# --------------------------------------------------------------------- passes
def _bytes(data):
    return np.frombuffer(data, np.uint8)


def _proofs(s, parts):
    """The proofs, back to back, in the program's own buffer (their length depends on the queries drawn), zeros after."""
    n, out = 0, s["out"]
    for part in parts:
        out[n:n + len(part)] = _bytes(part)
        n += len(part)
    out[n:s["n"]] = 0
    s["n"] = n
    return {"length": n, "proofs": out}


def _prove(s):
    c = s["case"]
    mode = G.INPUT_HOST if c["host"] else G.INPUT_SEEDED
    more = dict(seed=s["seed"], input_mode=mode, host_inputs=s.get("inputs"), config=s["config"],
                merkle_channel=c["channel"])
    if c["air"] == "poseidon":
        return _proofs(s, [G.prove_poseidon(c["log"], **more)])
    return _proofs(s, [G.prove_wide_fibonacci(c["log"], c["cols"], **more)])


def _serve(s):
    ids = [s["server"].submit(S.WIDE_FIBONACCI, log, cols, seed) for log, cols, seed in s["jobs"]]
    return _proofs(s, [s["server"].wait(i)[0] for i in ids])


def _plan(s):
    return _bytes(s["plan"].run(s["columns"]))


def _lde(s):
    """The trace's evaluations to coefficients (in place), then onto the larger domain."""
    trace, evals = list(s["trace"]), list(s["evals"])
    B.interpolate_columns(trace, s["log"], s["tw"])
    B.evaluate_polynomials(trace, s["out_log"], s["tw"], out=evals)
    return {"coeffs": s["trace"], "evals": s["evals"]}


def _merkle(s):
    B.commit_on_layer(s["log"], None, list(s["columns"]), out=s["layers"][-1])
    B.commit_node_layers(s["layers"])
    return s["layers"]


def _worklist(s):
    B.fft_worklist([("interpolate", a, b) for t, c in zip(s["traces"], s["coeffs"]) for a, b in zip(t, c)], s["tw"])
    B.fft_worklist([("evaluate", a, b) for c, e in zip(s["coeffs"], s["evals"]) for a, b in zip(c, e)], s["tw"])
    trees = B.merkle_worklist([list(e) for e in s["evals"]])
    return {"coeffs": torch.cat([c.view(-1) for c in s["coeffs"]]), "evals": torch.cat([e.view(-1) for e in s["evals"]]),
            "layers": torch.cat([t for layers in trees for t in layers])}


def _challenge(root):
    """A QM31 challenge from a Merkle root."""
    words = np.frombuffer(hashlib.blake2s(root).digest(), np.uint32)[:4]
    return [int(w) % P for w in words]


def _commit_layers(leaves, log):
    layers = [torch.empty(8 << k, dtype=torch.int32, device="cuda") for k in range(log)] + [leaves]
    B.commit_node_layers(layers)
    return B.batch_get_hashes(layers[0], [0]).tobytes()


def _fri(s):
    """The quotient's circle evaluation folded to a line, then every line layer committed and folded."""
    log = s["log"] - 1
    line = list(torch.zeros(4, 1 << log, dtype=torch.int32, device="cuda"))
    leaves = torch.empty(8 << log, dtype=torch.int32, device="cuda")
    B.fold_circle_into_line(line, list(s["planes"]), s["log"], s["alpha"], s["tw"], leaf_hashes=leaves)
    roots, first = [], torch.stack(line)
    while log > 1:
        roots.append(_commit_layers(leaves, log))
        leaves = torch.empty(8 << (log - 1), dtype=torch.int32, device="cuda")
        line = B.fold_line(line, log, _challenge(roots[-1]), s["tw"], leaf_hashes=leaves)
        log -= 1
    return {"first": first, "last": torch.stack(line), "roots": _bytes(b"".join(roots))}


def _deep(s):
    values = B.batch_eval_at_point(list(s["coeffs"]), s["point"])
    n = len(s["b"])
    partial = B.accumulate_numerators(list(s["evals"]), s["log"] + 1, range(n), s["b"], s["c"])
    quotient = B.compute_quotients_and_combine([(partial, s["log"] + 1, s["first"], s["point"])], s["log"] + 1)
    return {"values": np.array(values, np.uint32), "partial": torch.stack(partial), "quotient": torch.stack(quotient)}


_RUN = {"prove": _prove, "serve": _serve, "plan": _plan, "lde": _lde, "merkle": _merkle, "worklist": _worklist,
        "fri": _fri, "deep": _deep}


def run(state):
    return _RUN[state["kind"]](state)


# ----------------------------------------------------------------------- work
# 32-bit integer operations of the units of work: a radix-2 butterfly (one
# product, two sums, each reduced), a Blake2s compression (80 G functions of 12
# operations), a Poseidon252 permutation (107 cubes of two 8 x 8-limb products
# with their reductions), a QM31 x M31 multiply-add.
BUTTERFLY, COMPRESSION, PERMUTATION, QM_TERM = 7, 960, 214 * 160, 8


def _fft_ops(cols, log, out_log):
    return BUTTERFLY * cols * log * (1 << out_log) / 2


def _tree_ops(cols, log, felt=False):
    if felt:
        return PERMUTATION * (1 << log) * (((cols + 7) // 8) / 2 + 1 + 1)
    return COMPRESSION * (1 << log) * ((cols + 15) // 16 + 1)


def _proof_ops(air, log, cols, blowup, felt=False):
    expand = 2 if air == "poseidon" else 1
    ev = log + blowup
    ops = _fft_ops(cols, log, log) + _fft_ops(cols, log, ev) + _tree_ops(cols, ev, felt)
    if expand != blowup:
        ops += _fft_ops(cols, log, log + expand)
    ops += (1 << (log + expand)) * (8000 if air == "poseidon" else 24 * cols)  # constraints
    ops += QM_TERM * cols * ((1 << log) + (1 << ev))  # out-of-domain values, quotient numerators
    return ops + 3 * _tree_ops(4, ev, felt)  # composition and FRI trees


def work(case):
    """Bytes: each input read once and each output written once. `flops`:
    the 32-bit integer operations of the method (no floating point is used)."""
    kind = case["kind"]
    if kind == "prove":
        n_in = (16 if case["air"] == "poseidon" else 2) << case["log"]
        ops = _proof_ops(case["air"], case["log"], case["cols"], case["blowup"], case["channel"] == "poseidon252")
        size = case["queries"] * (4 * case["cols"] + 16 * (case["log"] + 3) ** 2) + 1000
        return {"bytes": 4 * n_in + size, "flops": ops}
    if kind == "serve":
        jobs = _jobs(case)
        return {"bytes": sum((8 << log) + 70 * (4 * cols + 16 * (log + 3) ** 2) for log, cols in jobs),
                "flops": sum(_proof_ops("wide_fibonacci", log, cols, 1) for log, cols in jobs)}
    if kind == "plan":
        logs, b = _plan_logs(case), case["blowup"]
        total, ops = sum(1 << k for k in logs), sum(_fft_ops(1, k, k) + _fft_ops(1, k, k + b) for k in logs)
        ops += COMPRESSION * ((2 << (max(logs) + b)) + (total << b) / 16)
        return {"bytes": 4 * total * (1 + 1 + (1 << b)) + (64 << (max(logs) + b)), "flops": ops}
    if kind == "lde":
        n, out = case["cols"] << case["log"], case["cols"] << (case["log"] + case["blowup"])
        return {"bytes": 4 * (2 * n + out), "flops": _fft_ops(case["cols"], case["log"], case["log"]) +
                _fft_ops(case["cols"], case["log"], case["log"] + case["blowup"])}
    if kind == "merkle":
        return {"bytes": (4 * case["cols"] + 64) << case["log"], "flops": _tree_ops(case["cols"], case["log"])}
    if kind == "worklist":
        c, logs = case["cols"], _tree_logs(case)
        return {"bytes": sum((4 * c * 4 << k) + (128 << k) for k in logs),
                "flops": sum(_fft_ops(c, k, k) + _fft_ops(c, k, k + 1) + _tree_ops(c, k + 1) for k in logs)}
    if kind == "fri":
        n = 1 << case["log"]  # source planes, every line layer's planes and its tree
        return {"bytes": 16 * n + 16 * n + 64 * n, "flops": 2 * COMPRESSION * n + 120 * n}
    n = case["cols"] << case["log"]
    return {"bytes": 4 * n + 8 * n + (2 * 32 << case["log"]), "flops": QM_TERM * 3 * n + (400 << case["log"])}


def tolerance(case):
    """Field elements, hashes and proof bytes: every correct implementation gives the same ones."""
    return "exact"


def exact(case, seed):
    """No output is a rounded number: whole values and bytes are compared as they are."""
    return None

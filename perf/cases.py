"""The workloads that the library is timed on, and the sizes it has to serve.

Every result is exact field arithmetic or a hash, so two correct
implementations agree to the last word: every case's tolerance is "exact".
``work`` counts each input and output word once, and the integer operations
that no implementation of the path can leave out: 3 field operations per
butterfly (one product, one sum, one difference), 1120 32-bit operations per
Blake2s compression, 8 per QM31 x M31 multiply-add (4 products, 4 sums) and 16
per QM31 product.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "stwo-metal_b200"))

from stwo_b200 import (B200Backend, Committer, ProveServer, SecureColumn, SeededFriProver, WideFibProver,  # noqa: E402
                       canonic_half_coset, wide_fib_config)

P = (1 << 31) - 1
COMPRESSION = 1120


class Column:
    """A column in the caller's own device memory."""

    def __init__(self, words):
        self.words = words
        self.ptr = words.data_ptr()
        self.length = words.numel()
        self.nbytes = 4 * self.length

    @property
    def log_size(self):
        return self.length.bit_length() - 1


class _Words:
    def __init__(self, buf, n):
        self.buf = buf
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (buf.ptr, False), "version": 3}


def words_of(buf):
    """A library buffer as a tensor, without a copy; it keeps the buffer."""
    return torch.as_tensor(_Words(buf, buf.nbytes // 4), device="cuda")


def slab(logs, values=None):
    """Columns of 2^log words side by side in one allocation."""
    words = torch.zeros(sum(1 << g for g in logs), dtype=torch.int32, device="cuda") if values is None else values
    cols, at = [], 0
    for g in logs:
        cols.append(Column(words[at:at + (1 << g)]))
        at += 1 << g
    return words, cols


def field_words(n, gen):
    return torch.randint(0, P, (n,), dtype=torch.int32, device="cuda", generator=gen)


def rngs(seed):
    return torch.Generator(device="cuda").manual_seed(seed), np.random.default_rng(seed)


def tree_for(be, log_domain):
    return be.precompute_twiddles(*canonic_half_coset(log_domain))


def uneven_logs(case):
    """The column sizes of a mixed commitment: uniform over [lo, hi]."""
    r = np.random.default_rng(case["shape_seed"])
    return [int(v) for v in r.integers(case["lo"], case["hi"] + 1, case["cols"])]


def requests(case):
    """Proof requests of a serving stream: 64 to 256 columns, log sizes lo..hi."""
    r = np.random.default_rng(case["shape_seed"])
    return [(int(r.integers(case["lo"], case["hi"] + 1)), int(r.integers(64, 257))) for _ in range(case["requests"])]


def listed():
    return [
        # a minimal proof: a caller's unit of latency, all launches and dependent steps
        {"name": "prove_small", "kind": "prove", "log": 10, "cols": 16, "blowup": 1, "queries": 3, "m31": True,
         "host": False},
        # the headline proof: 100 columns of 2^20 rows, default configuration
        {"name": "prove_wide", "kind": "prove", "log": 20, "cols": 100, "blowup": 1, "queries": 3, "m31": False,
         "host": False},
        # a mid-size proof of an odd width whose inputs come from pinned host memory
        {"name": "prove_host", "kind": "prove", "log": 17, "cols": 173, "blowup": 1, "queries": 3, "m31": False,
         "host": True},
        # the plain commitment: 32 natural-order columns of 2^16, blowup 1
        {"name": "commit_plain", "kind": "commit_plain", "log": 16, "cols": 32, "blowup": 1, "m31": False},
        # the mixed-degree commitment: 512 columns of 2^12..2^22, blowup 2
        {"name": "commit_uneven", "kind": "commit_uneven", "lo": 12, "hi": 22, "cols": 512, "blowup": 2, "m31": False,
         "shape_seed": 3},
        # a backend's trait calls one by one (bit reversal, interpolation, evaluation), an odd number of columns
        {"name": "lde_trait", "kind": "lde", "log": 19, "cols": 37, "blowup": 2},
        # sums of secure columns of every size from 2^12 to 2^20 (the composition accumulator)
        {"name": "accumulate", "kind": "accumulate", "lo": 12, "hi": 20},
        # FRI commitment and 70 openings of one secure column of 2^24
        {"name": "fri_heavy", "kind": "fri", "log": 24, "queries": 70, "m31": False},
        # stand-alone folds of a secure column of 2^20 down to one value, two layers a call
        {"name": "fold_chain", "kind": "fold", "log": 20, "step": 2},
        # FRI quotients of 100 columns of 2^20 opened at one point, a few of them at a second
        {"name": "quotients", "kind": "quotients", "log": 20, "cols": 100, "shifted": 7},
        # out-of-domain values of 108 polynomials of 2^20 coefficients
        {"name": "oods", "kind": "oods", "log": 20, "cols": 108},
        # a burst of proof requests at a resident server
        {"name": "serving", "kind": "serving", "lo": 14, "hi": 18, "requests": 8, "shape_seed": 11},
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _cols_under(rng, log, lo, hi, cells):
    return _log_uniform(rng, lo, max(lo, min(hi, cells >> log)))


def draw(rng):
    kind = rng.choice(["prove", "prove", "commit_plain", "commit_uneven", "lde", "lde", "accumulate", "fri", "fold",
                       "quotients", "oods", "serving"])
    if kind == "prove":
        log = rng.randint(8, 20)
        return {"kind": kind, "log": log, "cols": _cols_under(rng, log, 5, 256, 100 << 20),
                "blowup": rng.choice([1, 1, 2]) if log < 19 else 1, "queries": rng.choice([3, 3, 20, 70]),
                "m31": rng.random() < 0.25, "host": rng.random() < 0.4}
    if kind == "commit_plain":
        log = rng.randint(6, 21)
        return {"kind": kind, "log": log, "cols": _cols_under(rng, log, 1, 300, 64 << 20), "blowup": rng.choice([1, 2]),
                "m31": rng.random() < 0.25}
    if kind == "commit_uneven":
        lo = rng.randint(5, 14)
        return {"kind": kind, "lo": lo, "hi": rng.randint(lo, 20), "cols": _log_uniform(rng, 5, 400),
                "blowup": rng.choice([1, 2]), "m31": rng.random() < 0.25, "shape_seed": rng.randint(0, 1 << 30)}
    if kind == "lde":
        log = rng.randint(5, 22)
        return {"kind": kind, "log": log, "cols": _cols_under(rng, log, 1, 300, 80 << 20),
                "blowup": rng.choice([0, 1, 1, 2])}
    if kind == "accumulate":
        lo = rng.randint(4, 16)
        return {"kind": kind, "lo": lo, "hi": rng.randint(lo, 22)}
    if kind == "fri":
        return {"kind": kind, "log": rng.randint(8, 24), "queries": rng.choice([3, 20, 70]), "m31": rng.random() < 0.25}
    if kind == "fold":
        step = rng.randint(1, 3)
        return {"kind": kind, "log": rng.randint(6, 15 if step == 1 else 22), "step": step}
    if kind in ("quotients", "oods"):
        log = rng.randint(6, 22)
        case = {"kind": kind, "log": log, "cols": _cols_under(rng, log, 1, 300, 128 << 20)}
        if kind == "quotients":
            case["shifted"] = rng.randint(0, min(9, case["cols"]))
        return case
    lo = rng.randint(12, 16)
    return {"kind": kind, "lo": lo, "hi": rng.randint(lo, 18), "requests": rng.randint(2, 8),
            "shape_seed": rng.randint(0, 1 << 30)}


def prepare(case, seed):
    gen, rng = rngs(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind in ("prove", "serving", "fri"):
        s["proofs"] = [np.zeros(1 << 20, np.uint8) for _ in range(case.get("requests", 1))]
    if kind == "prove":
        cfg = wide_fib_config(case["log"], case["cols"], case["blowup"], n_queries=case["queries"],
                              m31_channel=case["m31"])
        s["prover"] = WideFibProver(cfg)
        n = 1 << case["log"]
        if case["host"]:
            pinned = [torch.from_numpy(rng.integers(0, P, n).astype(np.int32)).pin_memory() for _ in range(2)]
            s["pinned"] = pinned
            s["a"], s["b"] = (t.numpy().view(np.uint32) for t in pinned)
        else:
            s["a"], s["b"] = (Column(field_words(n, gen)) for _ in range(2))
        return s
    if kind == "serving":
        s["server"] = ProveServer(60 << 30, slots=3)
        s["requests"] = [(wide_fib_config(log, cols), rng.integers(0, P, 1 << log, dtype=np.uint32),
                          rng.integers(0, P, 1 << log, dtype=np.uint32)) for log, cols in requests(case)]
        # a running service has its provers resident: one burst of the same shapes on other inputs
        for t in [s["server"].submit(cfg, b, a) for cfg, a, b in s["requests"]]:
            s["server"].wait(t)
        return s
    be = s["be"] = B200Backend()
    if kind in ("commit_plain", "lde"):
        logs = [case["log"]] * case["cols"]
        big = [g + case["blowup"] for g in logs]
        s["tree"] = tree_for(be, case["log"] + case["blowup"] + 1)
        s["in"], s["in_cols"] = slab(logs, field_words(sum(1 << g for g in logs), gen))
        s["coef"], s["coef_cols"] = slab(logs)
        s["lde"], s["lde_cols"] = slab(big)
    elif kind == "commit_uneven":
        logs = uneven_logs(case)
        big = [g + case["blowup"] for g in logs]
        s["tree"] = tree_for(be, max(big) + 1)
        s["in"], s["in_cols"] = slab(logs, field_words(sum(1 << g for g in logs), gen))
        s["coef"], s["coef_cols"] = slab(logs)
        s["lde"], s["lde_cols"] = slab(big)
        s["layers"], s["layer_cols"] = slab([k + 3 for k in range(max(big) + 1)])
        s["committer"] = Committer(logs, case["blowup"], s["tree"], m31=case["m31"])
    elif kind == "accumulate":
        logs = list(range(case["lo"], case["hi"] + 1))
        s["cols"] = []
        for g in logs:
            s["cols"].append(SecureColumn(slab([g] * 4, field_words(4 << g, gen))[1]))
        s["other"] = SecureColumn(slab([case["hi"]] * 4, field_words(4 << case["hi"], gen))[1])
        s["out"], cols = slab([case["hi"]] * 4)
        s["sum"] = SecureColumn(cols)
    elif kind == "fri":
        s["tree"] = tree_for(be, case["log"] + 1)
        s["cols"] = slab([case["log"]] * 4, field_words(4 << case["log"], gen))[1]
        s["alphas"] = rng.integers(0, P, (case["log"], 4), dtype=np.uint32)
        s["at"] = np.sort(rng.integers(0, 1 << case["log"], case["queries"]).astype(np.uint64))
        s["prover"] = SeededFriProver(case["log"], s["tree"], m31=case["m31"])
    elif kind == "fold":
        s["tree"] = tree_for(be, case["log"] + 1)
        s["src"] = SecureColumn(slab([case["log"]] * 4, field_words(4 << case["log"], gen))[1])
        s["line"], cols = slab([case["log"] - 1] * 4)
        s["dst"] = SecureColumn(cols)
        s["alphas"] = rng.integers(0, P, (case["log"], 4), dtype=np.uint32)
    else:
        s["cols"] = slab([case["log"]] * case["cols"], field_words(case["cols"] << case["log"], gen))[1]
        s["point"] = rng.integers(1, P, 8, dtype=np.uint32)
        if kind == "quotients":
            def terms(k):
                return [(i, rng.integers(0, P, 4, dtype=np.uint32), rng.integers(0, P, 4, dtype=np.uint32))
                        for i in range(k)]
            s["batches"] = [(s["point"], terms(case["cols"]))]
            if case["shifted"]:
                s["batches"].append((rng.integers(1, P, 8, dtype=np.uint32), terms(case["shifted"])))
    return s


def _kept(s, proof, k=0):
    """A proof's bytes (their number depends on the queries it draws) in the caller's buffer, and their number."""
    out = s["proofs"][k]
    out[:len(proof)] = np.frombuffer(proof, dtype=np.uint8)
    return {"bytes": len(proof), "proof": out}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "prove":
        return _kept(s, (s["prover"].prove_host if case["host"] else s["prover"].prove)(s["a"], s["b"]))
    if kind == "serving":
        tickets = [s["server"].submit(cfg, a, b) for cfg, a, b in s["requests"]]
        return [_kept(s, s["server"].wait(t)[0], k) for k, t in enumerate(tickets)]
    if kind == "fri":
        return _kept(s, s["prover"].prove(s["cols"], s["alphas"], s["at"]))
    be = s["be"]
    if kind == "commit_plain":
        be.interpolate_natural_into(s["in_cols"], s["coef_cols"], s["tree"])
        be.evaluate_polynomials_into(s["coef_cols"], case["blowup"], s["tree"], s["lde_cols"])
        layers = be.build_merkle_layers(s["lde_cols"], case["log"] + case["blowup"], case["m31"])
        return {"coef": s["coef"], "lde": s["lde"], "layers": [words_of(b) for b in layers]}
    if kind == "commit_uneven":
        s["committer"].commit(s["in_cols"], s["coef_cols"], s["lde_cols"], s["layer_cols"])
        return {"coef": s["coef"], "lde": s["lde"], "layers": s["layers"]}
    if kind == "lde":
        be.bit_reverse_columns(s["in_cols"], s["coef_cols"])
        be.interpolate_columns(s["coef_cols"], s["tree"])
        be.evaluate_polynomials_into(s["coef_cols"], case["blowup"], s["tree"], s["lde_cols"])
        for c in s["lde_cols"][:4]:  # a few evaluations back to natural order, in place, one call each
            be.bit_reverse_column(c)
        return {"coef": s["coef"], "lde": s["lde"]}
    if kind == "accumulate":
        be.lift_and_accumulate(s["cols"], s["sum"])
        be.accumulate(s["sum"], s["other"])
        be.bit_reverse_secure_column(s["sum"])
        return s["out"]
    if kind == "fold":
        s["line"].zero_()
        be.fold_circle_into_line(s["dst"], s["src"], s["alphas"][0], s["tree"])
        ev, log, layers = s["dst"], case["log"] - 1, []
        while log > 0:
            step = min(case["step"], log)
            ev = be.fold_line(ev, s["alphas"][log], s["tree"], step)
            log -= step
            layers.append([words_of(c) for c in ev.cols])
        return {"line": s["line"], "layers": layers}
    if kind == "quotients":
        accs = be.accumulate_numerators(s["cols"], s["batches"])
        out = be.compute_quotients_and_combine(
            [(point, col, first) for (point, _), (col, first) in zip(s["batches"], accs)], case["log"])
        return {"partial": [[words_of(c) for c in col.cols] for col, _ in accs], "first": [f for _, f in accs],
                "quotients": [words_of(c) for c in out.cols]}
    return be.batch_eval_at_point(s["cols"], s["point"])


def _lde_work(logs, blowup):
    cells = sum(1 << g for g in logs)
    nbytes = 4 * cells * (2 + (1 << blowup))
    flies = sum((g << g) // 2 + (g << (g + blowup)) // 2 for g in logs)
    return nbytes, 3 * flies


def _tree_work(logs, lifting):
    """Bytes written and compressions of a lifted tree of columns of these log sizes."""
    logs = sorted(logs)
    tops = [max(logs[i:i + 16]) for i in range(0, len(logs), 16)]
    tops[-1] = lifting
    return 64 << lifting, sum(1 << t for t in tops) + (1 << lifting)


def _prove_work(log, cols, blowup):
    b, ops = _lde_work([log] * cols, blowup)
    big = log + blowup
    _, hashes = _tree_work([big] * cols, big)
    comp = 16 << big  # the composition's columns, the quotients and the FRI layers, 4 words a row each
    rows = cols << big
    # trace words are generated and coefficients and evaluations written; composition, OODS and quotients each
    # read the trace once more
    nbytes = b + 4 * rows * 2 + (4 * cols << log) + 64 * (3 << big) + 4 * comp
    return nbytes, ops + COMPRESSION * (hashes + (6 << big)) + 8 * (2 * rows + (cols << log)) + 4 * rows


def work(case):
    kind = case["kind"]
    if kind == "prove":
        b, o = _prove_work(case["log"], case["cols"], case["blowup"])
    elif kind == "serving":
        each = [_prove_work(log, cols, 1) for log, cols in requests(case)]
        b, o = sum(x for x, _ in each), sum(y for _, y in each)
    elif kind in ("commit_plain", "commit_uneven"):
        logs = [case["log"]] * case["cols"] if kind == "commit_plain" else uneven_logs(case)
        big = [g + case["blowup"] for g in logs]
        b, o = _lde_work(logs, case["blowup"])
        tb, h = _tree_work(big, max(big))
        b, o = b + tb, o + COMPRESSION * h
    elif kind == "lde":
        b, o = _lde_work([case["log"]] * case["cols"], case["blowup"])
        b += 8 * (min(4, case["cols"]) << (case["log"] + case["blowup"]))
    elif kind == "accumulate":
        b = 16 * (sum(1 << g for g in range(case["lo"], case["hi"] + 1)) + (2 << case["hi"]))
        o = 4 * sum(2 << g for g in range(case["lo"], case["hi"] + 1))
    elif kind == "fri":
        b, o = 64 * (2 << case["log"]) + (32 << case["log"]), (COMPRESSION * 4 + 40) << case["log"]
    elif kind == "fold":
        b, o = (16 + 8 + 24) << case["log"], 40 << case["log"]
    elif kind == "quotients":
        b = 4 * (case["cols"] << case["log"]) + 16 * ((2 if case["shifted"] else 1) + 1 << case["log"])
        o = 8 * ((case["cols"] + case["shifted"]) << case["log"])
    else:
        b, o = 4 * (case["cols"] << case["log"]), 8 * (case["cols"] << case["log"])
    return {"bytes": float(b), "flops": float(o)}


def tolerance(case):
    return "exact"

"""Performance cases: the prover's stages and whole proofs as a user of the framework runs them.

Every output is whole numbers (M31 words, Blake2s digests, proof words), so two correct runs on the
same inputs are equal word for word and `exact` has nothing to add. The "flops" of `work` are the
integer operations the path cannot do without: 3 per butterfly (one product, one sum, one
difference in M31), 1,120 per Blake2s compression (80 G steps of 14 operations), 1 per M31 product
or sum in the QM31 stages.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from proving_gb300 import gkr
from proving_gb300 import prover
from proving_gb300.backend import BaseColumn, CudaBackend, SecureColumnByCoords, canonic_half_coset
from proving_gb300.synthetic import mixed_trace_shape, seeded_log_sizes

P = (1 << 31) - 1
BLAKE_OPS = 1120
QM31_MUL_OPS = 28  # 16 products, 12 sums
FRI = (10, 1, 0, 70)  # pow bits, log blowup, log last layer degree bound, queries


def listed() -> list:
    return [
        # one FRI fold of a small layer (the reference's fri bench, 2^12 values): a single launch,
        # the latency a caller sees who drives FRI layer by layer
        {"name": "fold_line_2^12", "kind": "fold_line", "log_size": 12, "folds": 1},
        # the fold chain of a whole FRI layer stack of a 2^22 quotient column, as the commit-stage
        # benchmark runs it: circle into line, then every line fold in one call
        {"name": "fri_folds_2^22", "kind": "fri_folds", "log_size": 22},
        # the reference's fft bench: one long column, to coefficients and onto a twice larger domain
        {"name": "fft_1x2^24", "kind": "fft", "n_cols": 1, "log_size": 24, "log_blowup": 1},
        # the reference's merkle bench: 256 columns of 2^16 rows, leaves and all node layers
        {"name": "merkle_256x2^16", "kind": "merkle", "n_cols": 256, "log_size": 16},
        # the reference's pcs bench: 16 polynomials of 2^20 committed at blowup 1 (interpolate,
        # extend, lifted Merkle tree)
        {"name": "commit_16x2^20", "kind": "commit", "n_cols": 16, "log_size": 20, "log_blowup": 1},
        # the commit stage of the headline benchmark: a wide trace at blowup 2 (1 GiB of inputs)
        {"name": "commit_256x2^20", "kind": "commit", "n_cols": 256, "log_size": 20, "log_blowup": 2},
        # a ragged trace: columns of many sizes lifted into one tree, odd counts per size
        {"name": "commit_ragged_150", "kind": "commit_ragged", "n_cols": 150, "log_min": 9, "log_max": 20,
         "log_mean": 14.5, "shape_seed": 7, "log_blowup": 1},
        # out-of-domain sampling and the DEEP quotients of one size group of a proof
        {"name": "quotients_64x2^20", "kind": "quotients", "n_cols": 64, "log_size": 20, "log_blowup": 1},
        # GKR lookups: a generic LogUp instance batched with a grand product
        {"name": "gkr_2^22_2^20", "kind": "gkr", "lookup": "generic", "log_lookup": 22, "log_product": 20},
        # the smallest whole proof the serving loop sees often: Wide-Fibonacci 100 x 2^14
        {"name": "prove_wide_fib_100x2^14", "kind": "prove_wide_fib", "n_cols": 100, "log_size": 14},
        # the constraint side of a Poseidon2 proof (8 permutations a row, 1264 + 32 columns): the LogUp
        # interaction trace, then the constraint quotients on the four times larger domain
        {"name": "poseidon_constraints_2^16", "kind": "poseidon_constraints", "log_size": 16},
        # a mixed-size proof: 480 Wide-Fibonacci columns and 120 LogUp columns, log sizes 10..22
        {"name": "prove_mixed_600", "kind": "prove_mixed", "n_base": 600, "n_lookups": 120, "log_min": 10,
         "log_max": 22, "log_mean": 16.0, "shape_seed": 7},
    ]


def _log_uniform(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["fold_line", "fri_folds", "fft", "merkle", "commit", "commit", "commit_ragged", "quotients",
                       "gkr", "poseidon_constraints", "prove_wide_fib", "prove_mixed"])
    if kind == "fold_line":
        log_size = rng.randint(4, 22)
        return {"kind": kind, "log_size": log_size, "folds": rng.randint(1, min(log_size - 1, 12))}
    if kind == "fri_folds":
        return {"kind": kind, "log_size": rng.randint(5, 23)}
    if kind == "fft":
        log_size = rng.randint(6, 24)
        return {"kind": kind, "n_cols": _log_uniform(rng, 1, min(64, 1 << max(1, 26 - log_size))),
                "log_size": log_size, "log_blowup": rng.randint(0, 2)}
    if kind == "merkle":
        log_size = rng.randint(6, 20)
        return {"kind": kind, "n_cols": _log_uniform(rng, 1, min(700, 1 << (28 - log_size))), "log_size": log_size}
    if kind == "commit":
        log_size = rng.randint(6, 21)
        return {"kind": kind, "n_cols": _log_uniform(rng, 1, min(300, 1 << (28 - log_size))), "log_size": log_size,
                "log_blowup": rng.randint(1, 2)}
    if kind == "commit_ragged":
        log_min = rng.randint(5, 12)
        log_max = rng.randint(log_min + 2, 20)
        return {"kind": kind, "n_cols": _log_uniform(rng, 3, 300), "log_min": log_min, "log_max": log_max,
                "log_mean": round(log_min + (log_max - log_min) * rng.uniform(0.25, 0.6), 2),
                "shape_seed": rng.randint(1, 1000), "log_blowup": rng.randint(1, 2)}
    if kind == "quotients":
        log_size = rng.randint(8, 21)
        return {"kind": kind, "n_cols": _log_uniform(rng, 1, min(300, 1 << (27 - log_size))), "log_size": log_size,
                "log_blowup": rng.randint(1, 2)}
    if kind == "gkr":
        return {"kind": kind, "lookup": rng.choice(["generic", "multiplicities", "singles"]),
                "log_lookup": rng.randint(5, 22), "log_product": rng.randint(4, 21)}
    if kind == "prove_wide_fib":
        log_size = rng.randint(6, 20)
        return {"kind": kind, "n_cols": _log_uniform(rng, 3, min(250, 1 << (27 - log_size))), "log_size": log_size}
    if kind == "poseidon_constraints":
        return {"kind": kind, "log_size": rng.randint(4, 17)}
    log_min = rng.randint(6, 11)
    log_max = rng.randint(log_min + 3, 21)
    return {"kind": "prove_mixed", "n_base": _log_uniform(rng, 20, 500), "n_lookups": rng.randint(2, 16),
            "log_min": log_min, "log_max": log_max,
            "log_mean": round(log_min + (log_max - log_min) * rng.uniform(0.3, 0.55), 2),
            "shape_seed": rng.randint(1, 1000)}


def _ragged_logs(case) -> list:
    """The columns' log sizes, one column at least of the largest."""
    logs = [int(v) for v in seeded_log_sizes(case["shape_seed"], case["n_cols"], case["log_min"], case["log_max"],
                                             case["log_mean"])]
    logs[0] = case["log_max"]
    return logs


def _mixed_shape(case):
    return mixed_trace_shape(case["shape_seed"], case["n_base"], case["n_lookups"], case["log_min"], case["log_max"],
                             case["log_mean"])


class _Random:
    """Uniform M31 words on the device and QM31 challenges on the host, from the seed alone."""

    def __init__(self, seed: int):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.host = np.random.default_rng(seed)

    def block(self, n_cols: int, length: int) -> torch.Tensor:
        return torch.randint(0, P, (n_cols, length), dtype=torch.int32, device="cuda", generator=self.gen)

    def columns(self, n_cols: int, log_size: int) -> list:
        return BaseColumn.rows_of(self.block(n_cols, 1 << log_size))

    def secure(self, log_size: int) -> SecureColumnByCoords:
        return SecureColumnByCoords(self.columns(4, log_size))

    def felt(self) -> tuple:
        return tuple(int(v) for v in self.host.integers(0, P, 4))


def _empty(n_cols: int, log_size: int) -> torch.Tensor:
    return torch.empty((n_cols, 1 << log_size), dtype=torch.int32, device="cuda")


class _Group:
    """A trace's columns of one size with the blocks their coefficients and extension go to."""

    def __init__(self, rnd: _Random, n_cols: int, log_size: int, log_blowup: int):
        self.columns, self.log_ext = rnd.columns(n_cols, log_size), log_size + log_blowup
        self.coeff_block, self.ext_block = _empty(n_cols, log_size), _empty(n_cols, self.log_ext)
        self.coeffs, self.ext = BaseColumn.rows_of(self.coeff_block), BaseColumn.rows_of(self.ext_block)


def _twiddles(log_domain: int):
    return CudaBackend.precompute_twiddles(canonic_half_coset(log_domain))


class _ProofWords:
    """A buffer for a proof's words, zero beyond its end: the witness of another set of queries has
    another length."""

    def __init__(self, n_cols: int, height: int):
        self.words = np.zeros(4096 + FRI[3] * (n_cols + (height + 4) * (8 * height + 8)), np.int64)
        self.used = 0

    def fill(self, proof: bytes) -> np.ndarray:
        w = np.frombuffer(proof, dtype="<u8")
        self.words[:w.size] = w
        self.words[w.size:max(w.size, self.used)] = 0
        self.used = w.size
        return self.words


def _flat(felts) -> np.ndarray:
    """The words of nested lists of field elements."""
    out, stack = [], [felts]
    while stack:
        x = stack.pop()
        if isinstance(x, (list, tuple)):
            stack.extend(reversed(x))
        else:
            out.append(int(x))
    return np.asarray(out, np.int64)


def prepare(case, seed):
    rnd = _Random(seed)
    kind = case["kind"]
    if kind == "fold_line":
        n = case["log_size"]
        return {"kind": kind, "values": rnd.secure(n), "alphas": [rnd.felt() for _ in range(case["folds"])],
                "twiddles": _twiddles(n + 1)}
    if kind == "fri_folds":
        n = case["log_size"]
        return {"kind": kind, "values": rnd.secure(n), "alphas": [rnd.felt() for _ in range(n)],
                "twiddles": _twiddles(n)}
    if kind in ("fft", "commit"):
        n, b = case["log_size"], case["log_blowup"]
        return {"kind": kind, "groups": [_Group(rnd, case["n_cols"], n, b)], "height": n + b,
                "twiddles": _twiddles(n + b)}
    if kind == "merkle":
        return {"kind": kind, "columns": rnd.columns(case["n_cols"], case["log_size"]), "log_size": case["log_size"]}
    if kind == "commit_ragged":
        b, logs = case["log_blowup"], _ragged_logs(case)
        return {"kind": kind, "groups": [_Group(rnd, logs.count(n), n, b) for n in sorted(set(logs))],
                "height": case["log_max"] + b, "twiddles": _twiddles(case["log_max"] + b)}
    if kind == "quotients":
        n, c, b = case["log_size"], case["n_cols"], case["log_blowup"]
        point = prover.random_point(rnd.felt())
        return {"kind": kind, "columns": rnd.columns(c, n), "point": point,
                "coeffs": np.asarray([[rnd.felt() for _ in range(3)] for _ in range(c)], np.uint32),
                "log_size": n, "log_blowup": b, "twiddles": _twiddles(n)}
    if kind == "gkr":
        n, m = case["log_lookup"], case["log_product"]
        den = gkr.Mle(rnd.block(4, 1 << n), n)
        if case["lookup"] == "generic":
            lookup = gkr.Layer(gkr.LOGUP_GENERIC, [gkr.Mle(rnd.block(4, 1 << n), n), den])
        elif case["lookup"] == "multiplicities":
            lookup = gkr.Layer(gkr.LOGUP_MULTIPLICITIES, [gkr.Mle(rnd.block(1, 1 << n), n, base=True), den])
        else:
            lookup = gkr.Layer(gkr.LOGUP_SINGLES, [den])
        product = gkr.Layer(gkr.GRAND_PRODUCT, [gkr.Mle(rnd.block(4, 1 << m), m)])
        return {"kind": kind, "layers": [lookup, product]}
    if kind == "prove_wide_fib":
        n = case["log_size"]
        a, b = rnd.columns(2, n)
        return {"kind": kind, "a": a, "b": b, "n_cols": case["n_cols"], "log_size": n, "twiddles": _twiddles(n + 2),
                "words": _ProofWords(case["n_cols"] + 8, n + 1)}
    if kind == "poseidon_constraints":
        n, c, i = case["log_size"], CudaBackend.POSEIDON_COLS, CudaBackend.POSEIDON_INTERACTION_COLS
        return {"kind": kind, "trace": rnd.columns(c, n), "trace_evals": rnd.columns(c, n + 2),
                "inter_evals": rnd.columns(i, n + 2), "log_size": n, "lookup": rnd.felt() + rnd.felt(),
                "rc": rnd.host.integers(0, P, (CudaBackend.POSEIDON_CONSTRAINTS, 4)).astype(np.uint32)}
    comps, lookup_logs = _mixed_shape(case)
    top = max([n for _, n in comps] + lookup_logs)
    return {"kind": kind, "comps": comps, "seeds": [rnd.columns(2, n) for _, n in comps], "lookup_logs": lookup_logs,
            "lookups": [rnd.columns(1, n)[0] for n in lookup_logs], "twiddles": _twiddles(top + 2),
            "words": _ProofWords(sum(n for n, _ in comps) + 6 * len(lookup_logs) + 8, top + 1)}


def run(state):
    kind, B = state["kind"], CudaBackend
    if kind == "fold_line":
        return [c.data for c in B.fold_line(state["values"], state["alphas"], state["twiddles"]).columns]
    if kind == "fri_folds":
        line = B.fold_circle_into_line(state["values"], state["alphas"][0], state["twiddles"])
        last = B.fold_line(line, state["alphas"][1:], state["twiddles"])
        return [c.data for c in line.columns + last.columns]
    if kind in ("fft", "commit", "commit_ragged"):
        groups, tw = state["groups"], state["twiddles"]
        for g in groups:
            B.interpolate_columns_into(g.columns, tw, g.coeffs)
        for g in groups:
            B.evaluate_polynomials(g.coeffs, g.log_ext, tw, g.ext)
        out = [b for g in groups for b in (g.coeff_block, g.ext_block)]
        if kind != "fft":
            out.append(B.merkle_commit([c for g in groups for c in g.ext], state["height"]).all)
        return out
    if kind == "merkle":
        return [B.merkle_commit(state["columns"], state["log_size"]).all]
    if kind == "quotients":
        weights = B.barycentric_weights(state["log_size"], state["point"])
        sampled = B.barycentric_eval_at_point(state["columns"], weights)
        part, first = B.accumulate_numerators(state["columns"], state["coeffs"], state["log_blowup"])
        q = B.compute_quotients_and_combine([part], [state["point"]], [first], state["log_size"],
                                            state["log_blowup"], state["twiddles"])
        return [sampled, first.astype(np.int64)] + [c.data for c in part.columns + q.columns]
    if kind == "gkr":
        channel = prover.Blake2sChannel()
        proof, artifact = gkr.prove_batch_native(channel, state["layers"])
        masks = [m.columns for inst in proof.layer_masks_by_instance for m in inst]
        claims = proof.output_claims_by_instance + artifact.claims_to_verify_by_instance
        return [_flat(proof.sumcheck_proofs), _flat(masks), _flat(claims), _flat(artifact.ood_point),
                np.frombuffer(channel.digest, np.uint8)]
    if kind == "prove_wide_fib":
        trace = B.wide_fib_trace(state["a"], state["b"], state["n_cols"])
        return state["words"].fill(B.prove_wide_fib_native([trace], [state["log_size"]], FRI, state["twiddles"]))
    if kind == "poseidon_constraints":
        inter, claimed = B.poseidon_interaction(state["trace"], state["lookup"])
        accum = SecureColumnByCoords.zeros(4 << state["log_size"])
        B.poseidon_composition(state["trace_evals"], state["inter_evals"], state["log_size"], state["lookup"], claimed,
                               state["rc"], accum)
        return [c.data for c in inter + accum.columns] + [claimed.astype(np.int64)]
    traces = [B.wide_fib_trace(a, b, n) for (a, b), (n, _) in zip(state["seeds"], state["comps"])]
    proof, claimed = B.prove_fib_and_lookups_native(traces, [n for _, n in state["comps"]], state["lookups"],
                                                    state["lookup_logs"], FRI, state["twiddles"])
    return [state["words"].fill(proof), np.asarray(claimed, np.int64)]


def _butterflies(n_cols: int, layers: int, log_size: int) -> int:
    return n_cols * layers << max(log_size - 1, 0)


def _tree_work(logs, height: int):
    """Compressions of a lifted tree: each block of 16 columns once at the size that determines it."""
    logs = sorted(logs)
    blocks = max(1, (len(logs) + 15) // 16)
    at = [logs[min(16 * b + 15, len(logs) - 1)] for b in range(blocks - 1)] + [height]
    return sum(1 << n for n in at) + (1 << height)


def _commit_work(logs, log_blowup: int, height: int) -> dict:
    words = sum(1 << n for n in logs)
    ext = words << log_blowup
    fly = sum(_butterflies(1, n, n) + _butterflies(1, n, n + log_blowup) for n in logs)
    tree = _tree_work([n + log_blowup for n in logs], height)
    return {"bytes": 4 * (2 * words + ext) + (64 << height), "flops": 3 * fly + BLAKE_OPS * tree}


def _proof_work(groups, log_blowup: int, height: int, inputs: int) -> dict:
    """groups: (columns, log size) committed. The bytes are the inputs alone, since a proof is a few
    hundred kilobytes and every other array is the prover's own; the operations are the committed
    columns' transforms, trees, samples and numerators and the FRI layers' trees."""
    logs = [n for c, n in groups for _ in range(c)]
    w = _commit_work(logs, log_blowup, height)
    ext = sum(1 << (n + log_blowup) for n in logs)
    return {"bytes": inputs + (1 << 18), "flops": w["flops"] + 16 * ext + 2 * BLAKE_OPS * (2 << height)}


def work(case) -> dict:
    kind = case["kind"]
    if kind == "fold_line":
        n, k = 1 << case["log_size"], case["folds"]
        return {"bytes": 16 * (n + (n >> k)) + 4 * n, "flops": (n - (n >> k)) * (QM31_MUL_OPS + 12)}
    if kind == "fri_folds":
        n = 1 << case["log_size"]
        return {"bytes": 16 * n + 16 * (n >> 1) + 16 + 4 * n, "flops": n * (QM31_MUL_OPS + 12)}
    if kind == "fft":
        n, c, b = case["log_size"], case["n_cols"], case["log_blowup"]
        return {"bytes": 4 * c * ((2 << n) + (1 << (n + b))),
                "flops": 3 * (_butterflies(c, n, n) + _butterflies(c, n, n + b))}
    if kind == "merkle":
        n, c = case["log_size"], case["n_cols"]
        return {"bytes": 4 * c * (1 << n) + (64 << n), "flops": BLAKE_OPS * _tree_work([n] * c, n)}
    if kind == "commit":
        n, b = case["log_size"], case["log_blowup"]
        return _commit_work([n] * case["n_cols"], b, n + b)
    if kind == "commit_ragged":
        return _commit_work(_ragged_logs(case), case["log_blowup"], case["log_max"] + case["log_blowup"])
    if kind == "quotients":
        n, c, b = case["log_size"], case["n_cols"], case["log_blowup"]
        part = 1 << (n - b)
        return {"bytes": 4 * c * (1 << n) + 16 * part + (16 << n),
                "flops": c * (8 << n) + c * 8 * part + 3 * _butterflies(4, n - b, n - b) + 3 * _butterflies(4, n - b, n)}
    if kind == "gkr":
        n, m = 1 << case["log_lookup"], 1 << case["log_product"]
        per = {"generic": 32, "multiplicities": 20, "singles": 16}[case["lookup"]]
        return {"bytes": per * n + 16 * m, "flops": (n * 12 + m * 5) * QM31_MUL_OPS}
    if kind == "prove_wide_fib":
        n, c = case["log_size"], case["n_cols"]
        return _proof_work([(c, n), (8, n)], 1, n + 1, 8 << n)
    if kind == "poseidon_constraints":
        # per evaluation row 8 instances of 142 round constraints: a product by the constraint's QM31
        # weight (4 products, 4 sums) each, beside the permutation's own 142 x 3 products and its
        # matrices (about 16 x 30 sums)
        n = 1 << case["log_size"]
        return {"bytes": 4 * n * (1264 + 32) + 16 * n * (1264 + 32) + 64 * n,
                "flops": 4 * n * 8 * (142 * (8 + 3) + 22 * 16 * 8) + n * 8 * 40 * QM31_MUL_OPS // 4}
    comps, lookup_logs = _mixed_shape(case)
    top = max([n for _, n in comps] + lookup_logs)
    inputs = sum(8 << n for _, n in comps) + sum(4 << n for n in lookup_logs)
    return _proof_work(comps + [(5, n) for n in lookup_logs] + [(8, top)], 1, top + 1, inputs)


def exact(case, seed):
    """None: the outputs are whole numbers, which are compared for equality."""
    return None

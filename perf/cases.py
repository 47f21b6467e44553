"""The calls that a proof system makes of this framework, as cases to be timed.

A prover commits polynomials and traces (Reed-Solomon low-degree extension,
then a Poseidon2 Merkle tree), opens them (FRI, Basefold, the SP1 stacked open)
and now and then only encodes or only hashes. The cases are these calls, through
the package's public classes, from 2^10-coefficient polynomials to a 2^20-row
trace of 64 columns, over BabyBear with the built-in Poseidon2 instance and over
KoalaBear with SP1's and Plonky3's run-time instances. Verification runs on
hosts without a GPU and is not among them.

Every output is a field word, so `exact` speaks only where a plain 64-bit
restatement is short (the transforms); everywhere the words have to be equal.
"""

from __future__ import annotations

import json
import math
import os
import random

import numpy as np
import torch

from zorch_gb300.batch import BatchCommitter, MatrixJob
from zorch_gb300.coding import BitReversedReedSolomon, ReedSolomon
from zorch_gb300.commit import (MerkleTree, Poseidon2, SingleMatrixCommitmentScheme,
                                StridedMerkleTree)
from zorch_gb300.field import BABYBEAR, KOALABEAR, to_mont
from zorch_gb300.jagged import stacked_basefold_open, stacked_commit
from zorch_gb300.pcs import (BasefoldProver, FoldState, FriParams, FriProver,
                             PreFoldKGroupCommitRound, fold_rounds)
from zorch_gb300.stage import OpeningClaim, OpeningWitness
from zorch_gb300.transcript import DuplexTranscript

GOLDEN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests",
                      "golden")
FIELDS = {"babybear": BABYBEAR, "koalabear": KOALABEAR}


def listed():
    return [
        # one polynomial committed by itself: the smallest unit a prover asks
        # for, and the latency of a whole commit (2^16 coefficients, blowup 2)
        {"name": "commit_poly_2p16", "kind": "commit_polys", "count": 1, "log_k": 16,
         "log_blowup": 1},
        # a short, odd-width matrix (a preprocessed table): few leaves, wide blowup
        {"name": "commit_rows_2p13x37_b8", "kind": "commit_rows", "log_k": 13, "width": 37,
         "log_blowup": 3},
        # the trace commit of a STARK: 2^20 rows of 64 columns at blowup 4
        {"name": "commit_rows_2p20x64_b4", "kind": "commit_rows", "log_k": 20, "width": 64,
         "log_blowup": 2},
        # many tables of one machine committed together, heights and widths uneven
        {"name": "commit_batch_16_uneven", "kind": "commit_batch", "count": 16, "min_log_k": 12,
         "max_log_k": 18, "max_width": 128, "shape_seed": 5},
        # SP1's component commit over KoalaBear: bit-reversed code, column-major
        # leaves, the run-time Poseidon2 instance, an odd column count
        {"name": "smcs_koala_2p18x11_b4", "kind": "smcs_commit", "log_k": 18, "width": 11,
         "log_blowup": 2},
        # encode and FRI commit phase of one large polynomial, EF4 challenges,
        # down to 2^8, 100 queries
        {"name": "fri_phase_2p22", "kind": "fri_phase", "log_k": 22, "log_blowup": 1,
         "rounds": 15, "queries": 100, "limbs": 4},
        # a small FRI open of two committed polynomials (DEEP quotient, folds,
        # queries) at a base-field point: launches and latency
        {"name": "fri_open_2x2p12", "kind": "fri_open", "count": 2, "log_k": 12, "log_blowup": 2,
         "rounds": 10, "queries": 32, "limbs": 1, "point_limbs": 1},
        # Basefold open of a committed matrix at one EF4 point
        {"name": "basefold_open_2p20x8", "kind": "basefold_open", "log_k": 20, "width": 8,
         "log_blowup": 1, "queries": 64},
        # SP1's stacked open of two committed rounds with its proof of work
        {"name": "sp1_open_2p20_8_4", "kind": "sp1_open", "log_k": 20, "width": 8, "width2": 4,
         "log_blowup": 1, "queries": 64, "pow_bits": 16},
        # k-ary fold-and-commit rounds over KoalaBear (Plonky3's instance)
        {"name": "kary4_fold_2p22", "kind": "kary_fold", "log_n": 22, "log_arity": 2, "rounds": 2},
        # a query-strided tree over row-major rows (WHIR)
        {"name": "strided_2p20x8_16", "kind": "strided_commit", "log_h": 20, "width": 8,
         "rows_per_query": 16},
        # low-degree extension from evaluations (inverse transform, then the
        # coset transform) of a medium table with an odd column count
        {"name": "extend_2p16x99_b2", "kind": "extend", "field": "babybear", "log_k": 16,
         "width": 99, "log_blowup": 1},
    ]


def _log_uniform(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges, no larger than the trace commit."""
    cap = work(next(c for c in listed() if c["name"] == "commit_rows_2p20x64_b4"))
    while True:
        c = _draw(rng)
        w = work(c)
        if w["bytes"] <= cap["bytes"] and w["flops"] <= cap["flops"]:
            return c


def _draw(rng):
    kind = rng.choice(["commit_polys", "commit_rows", "commit_batch", "smcs_commit", "fri_phase",
                       "fri_open", "basefold_open", "sp1_open", "kary_fold", "strided_commit",
                       "extend"])
    c = {"kind": kind}
    if kind == "commit_polys":
        c.update(log_k=rng.randint(10, 20), count=rng.randint(1, 8), log_blowup=rng.randint(1, 3))
    elif kind in ("commit_rows", "smcs_commit"):
        lk = rng.randint(10, 20 if kind == "commit_rows" else 18)
        lb = rng.randint(1, 3)
        # at most 2^26 committed words
        cap = max(1, min(256, 1 << (26 - lk)))
        c.update(log_k=lk, width=_log_uniform(rng, 1, cap), log_blowup=min(lb, 2) if lk > 18 else lb)
    elif kind == "commit_batch":
        lo = rng.randint(10, 14)
        c.update(count=rng.randint(2, 24), min_log_k=lo, max_log_k=lo + rng.randint(1, 4),
                 max_width=rng.randint(8, 128), shape_seed=rng.randint(0, 1 << 20))
    elif kind == "fri_phase":
        lk = rng.randint(12, 22)
        lb = rng.randint(1, 2) if lk < 22 else 1
        c.update(log_k=lk, log_blowup=lb, rounds=max(1, lk + lb - rng.randint(6, 9)),
                 queries=rng.randint(20, 128), limbs=rng.choice([1, 4]))
    elif kind == "fri_open":
        lk = rng.randint(8, 16)
        lb = rng.randint(1, 2)
        c.update(count=rng.randint(1, 2), log_k=lk, log_blowup=lb, rounds=lk - rng.randint(0, 4),
                 queries=rng.randint(16, 100), limbs=rng.choice([1, 4]),
                 point_limbs=rng.choice([1, 4]))
    elif kind == "basefold_open":
        c.update(log_k=rng.randint(10, 20), width=_log_uniform(rng, 1, 48),
                 log_blowup=rng.randint(1, 2), queries=rng.randint(16, 100))
    elif kind == "sp1_open":
        c.update(log_k=rng.randint(10, 20), width=_log_uniform(rng, 1, 32),
                 width2=_log_uniform(rng, 1, 16), log_blowup=rng.randint(1, 2),
                 queries=rng.randint(16, 100), pow_bits=rng.randint(0, 16))
    elif kind == "kary_fold":
        la = rng.randint(1, 4)
        ln = rng.randint(14, 22)
        c.update(log_n=ln, log_arity=la, rounds=rng.randint(1, max(1, (ln - 8) // la)))
    elif kind == "strided_commit":
        c.update(log_h=rng.randint(12, 20), width=_log_uniform(rng, 1, 32),
                 rows_per_query=1 << rng.randint(0, 6))
    else:
        lk = rng.randint(8, 20)
        c.update(field=rng.choice(["babybear", "koalabear"]), log_k=lk,
                 width=_log_uniform(rng, 1, max(1, min(256, 1 << (25 - lk)))),
                 log_blowup=rng.randint(1, 3))
    return c


# ------------------------------------------------------------- inputs ----
def _words(gen, field, *shape):
    """Uniform field elements as words in [0, p)."""
    return torch.randint(0, field.p, shape, generator=gen, device="cuda", dtype=torch.int64).to(
        torch.int32)


def _instance(name):
    with open(os.path.join(GOLDEN, *name.split("/"))) as f:
        d = json.load(f)
    return Poseidon2.from_params(KOALABEAR, d["alpha"], d["external_initial"],
                                 d["external_terminal"], d["internal_rc"], d["internal_diag"],
                                 d.get("internal_j_scale", 1))


def _batch_shapes(case):
    r = random.Random(case["shape_seed"])
    return [(r.randint(1, case["max_width"]), r.randint(case["min_log_k"], case["max_log_k"]),
             r.randint(1, 3)) for _ in range(case["count"])]


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    kind = case["kind"]
    s = {"kind": kind, "case": dict(case)}
    if kind == "commit_polys":
        code = ReedSolomon(1 << case["log_k"], 1 << case["log_blowup"], BABYBEAR, coset_shift=31,
                           generator=31)
        s["prover"] = FriProver(FriParams(code, MerkleTree(Poseidon2.builtin(BABYBEAR)),
                                          1, 1, 4))
        s["polys"] = [_words(gen, BABYBEAR, 1 << case["log_k"]) for _ in range(case["count"])]
    elif kind == "commit_rows":
        code = ReedSolomon(1 << case["log_k"], 1 << case["log_blowup"], BABYBEAR, coset_shift=31,
                           generator=31)
        s["prover"] = BasefoldProver(code, MerkleTree(Poseidon2.builtin(BABYBEAR),
                                                      column_major=True))
        s["x"] = _words(gen, BABYBEAR, case["width"], 1 << case["log_k"])
    elif kind == "commit_batch":
        s["committer"] = BatchCommitter(Poseidon2.builtin(BABYBEAR), BABYBEAR)
        s["jobs"] = [MatrixJob(_words(gen, BABYBEAR, w, 1 << lk), lb)
                     for w, lk, lb in _batch_shapes(case)]
    elif kind == "smcs_commit":
        s["smcs"] = SingleMatrixCommitmentScheme(_instance("sp1_fibonacci/sp1_koalabear16.json"))
        s["code"] = BitReversedReedSolomon(1 << case["log_k"], 1 << case["log_blowup"], KOALABEAR)
        s["x"] = _words(gen, KOALABEAR, case["width"], 1 << case["log_k"])
    elif kind in ("fri_phase", "fri_open"):
        perm = Poseidon2.builtin(BABYBEAR)
        code = ReedSolomon(1 << case["log_k"], 1 << case["log_blowup"], BABYBEAR, coset_shift=31,
                           generator=31)
        s["code"], s["perm"] = code, perm
        s["prover"] = FriProver(FriParams(code, MerkleTree(perm), case["rounds"],
                                          case["queries"], case["limbs"]))
        if kind == "fri_phase":
            s["x"] = _words(gen, BABYBEAR, 1 << case["log_k"])
        else:
            polys = [_words(gen, BABYBEAR, 1 << case["log_k"]) for _ in range(case["count"])]
            roots, data = s["prover"].commit(polys)
            points = [_words(gen, BABYBEAR, case["point_limbs"]) for _ in polys]
            s["claim"], s["witness"] = OpeningClaim(roots, points), OpeningWitness(data)
    elif kind == "basefold_open":
        perm = Poseidon2.builtin(BABYBEAR)
        code = ReedSolomon(1 << case["log_k"], 1 << case["log_blowup"], BABYBEAR, coset_shift=31)
        s["perm"] = perm
        s["prover"] = BasefoldProver(code, MerkleTree(perm, column_major=True),
                                     num_queries=case["queries"])
        _, s["data"] = s["prover"].commit_columns(_words(gen, BABYBEAR, case["width"],
                                                         1 << case["log_k"]))
        s["z"] = _words(gen, BABYBEAR, case["log_k"], 4)
    elif kind == "sp1_open":
        s["perm"] = _instance("sp1_fibonacci/sp1_koalabear16.json")
        s["smcs"] = SingleMatrixCommitmentScheme(s["perm"])
        s["code"] = BitReversedReedSolomon(1 << case["log_k"], 1 << case["log_blowup"], KOALABEAR)
        s["rounds"] = [stacked_commit(s["smcs"], s["code"],
                                      _words(gen, KOALABEAR, w, 1 << case["log_k"]))
                       for w in (case["width"], case["width2"])]
        s["z"] = _words(gen, KOALABEAR, case["log_k"] + 2, 4)
        s["eval"] = _words(gen, KOALABEAR, 4)
    elif kind == "kary_fold":
        s["perm"] = _instance("koalabear16.json")
        k = 1 << case["log_arity"]
        s["code"] = ReedSolomon(1 << (case["log_n"] - 1), 2, KOALABEAR, fold_factor=k)
        s["tree"] = MerkleTree(s["perm"])
        s["cw"] = s["code"].encode(_words(gen, KOALABEAR, 1 << (case["log_n"] - 1)))
    elif kind == "strided_commit":
        s["tree"] = StridedMerkleTree(Poseidon2.builtin(BABYBEAR), case["rows_per_query"])
        s["x"] = _words(gen, BABYBEAR, 1 << case["log_h"], case["width"])
    else:
        field = FIELDS[case["field"]]
        s["code"] = ReedSolomon(1 << case["log_k"], 1 << case["log_blowup"], field,
                                coset_shift=field.generator)
        s["x"] = _words(gen, field, case["width"], 1 << case["log_k"])
    return s


def _opening(op):
    return [op.row, op.path]


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "commit_polys":
        # canonical coefficients, as a prover has them, then FriProver.commit
        roots, data = state["prover"].commit([to_mont(BABYBEAR, x) for x in state["polys"]])
        return [roots, [[c.codeword, c.digest_layers.flat] for c in data.polys]]
    if kind == "commit_rows":
        root, data = state["prover"].commit_columns(to_mont(BABYBEAR, state["x"]))
        return [root, data.codeword, data.digest_layers.flat]
    if kind == "commit_batch":
        return [[m.codeword, m.layers.flat] for m in state["committer"].commit(state["jobs"])]
    if kind == "smcs_commit":
        r = stacked_commit(state["smcs"], state["code"], state["x"])
        return [r.commitment, r.codeword, r.digest_layers.flat]
    if kind == "fri_phase":
        cw = state["code"].encode(to_mont(BABYBEAR, state["x"]))
        p, _, _ = state["prover"].commit_phase(cw, DuplexTranscript.new(state["perm"]))
        return [cw, p.roots, p.betas, p.final_layer, p.positions,
                [_opening(o) for o in p.openings]]
    if kind == "fri_open":
        r = state["prover"].prove(state["claim"], state["witness"],
                                  DuplexTranscript.new(state["perm"]))
        op = r.reduction_proof
        return [op.values, [p.parts() for p in op.proof], r.transcript.state]
    if kind == "basefold_open":
        values, p, t = state["prover"].open_batch([state["data"]], state["z"],
                                                  DuplexTranscript.new(state["perm"]))
        return [values, p.uni_msgs, p.fri_roots, p.final_poly, p.positions,
                [_opening(o) for o in p.component_openings],
                [_opening(o) for o in p.query_openings], t.state]
    if kind == "sp1_open":
        p, t = stacked_basefold_open(
            state["smcs"], state["code"], state["rounds"], state["z"], state["eval"],
            case["log_k"], num_queries=case["queries"], pow_bits=case["pow_bits"],
            transcript=DuplexTranscript.new(state["perm"]))
        return [p.fri_raw_roots, p.fri_commitments, p.univariate_messages, p.final_poly,
                p.pow_witness, p.batch_evals, [list(o) for o in p.component_openings],
                [list(o) for o in p.query_openings], p.positions]
    if kind == "kary_fold":
        st, t, roots = fold_rounds(PreFoldKGroupCommitRound(state["code"], state["tree"]),
                                   FoldState(state["cw"]), DuplexTranscript.new(state["perm"]),
                                   case["rounds"])
        return [st.codeword, roots, [[x.codeword, x.digest_layers.flat] for x in st.layers],
                t.state]
    if kind == "strided_commit":
        root, layers = state["tree"].commit(state["x"])
        return [root, layers.flat]
    return state["code"].extend(state["x"])


# --------------------------------------------------------------- work ----
# Integer operations counted: a modular product as 4 (the wide product, the two
# multiplies of its reduction, the subtract), a modular add as 2. One width-16
# permutation: BabyBear x^7, 8 full and 13 partial rounds; KoalaBear x^3, 8 and 20.
_PERM = {"babybear": (8 * 16 + 13) * 16 + 9 * 72 * 2 + 13 * 48 * 2,
         "koalabear": (8 * 16 + 20) * 8 + 9 * 72 * 2 + 20 * (31 * 2 + 16 * 4)}


def _tree(leaves, perms_per_leaf, field):
    """(bytes, ops): every digest written once, every permutation run once."""
    return 32 * (2 * leaves - 1), _PERM[field] * (leaves * perms_per_leaf + leaves - 1)


def _lde(width, log_k, log_b):
    n = width << (log_k + log_b)
    return 4 * ((width << log_k) + n), n * log_k // 2 * 8


def _sum(*pairs):
    return tuple(sum(p) for p in zip(*pairs))


def _folds(log_n, rounds, field, limbs):
    """Pair-leaf trees and folds of `rounds` layers from 2^log_n points."""
    total = (0, 0)
    for r in range(rounds):
        n = 1 << (log_n - r)
        total = _sum(total, _tree(n // 2, 1, field), (4 * limbs * (n + n // 2), n * 4 * limbs))
    return total


def work(case):
    kind = case["kind"]
    if kind == "commit_polys":
        n = 1 << (case["log_k"] + case["log_blowup"])
        one = _sum(_lde(1, case["log_k"], case["log_blowup"]), _tree(n // 2, 1, "babybear"))
        b, f = one[0] * case["count"], one[1] * case["count"]
    elif kind in ("commit_rows", "smcs_commit"):
        field = "babybear" if kind == "commit_rows" else "koalabear"
        b, f = _sum(_lde(case["width"], case["log_k"], case["log_blowup"]),
                    _tree(1 << (case["log_k"] + case["log_blowup"]), -(-case["width"] // 8),
                          field))
    elif kind == "commit_batch":
        b, f = _sum(*[_sum(_lde(w, lk, lb), _tree(1 << (lk + lb), -(-w // 8), "babybear"))
                      for w, lk, lb in _batch_shapes(case)])
    elif kind == "fri_phase":
        b, f = _sum(_lde(1, case["log_k"], case["log_blowup"]),
                    _folds(case["log_k"] + case["log_blowup"], case["rounds"], "babybear",
                           case["limbs"]))
    elif kind == "fri_open":
        n = 1 << (case["log_k"] + case["log_blowup"])
        one = _sum((4 << case["log_k"], 8 << case["log_k"]),
                   (4 * n * (1 + case["point_limbs"]), n * 3 * 16 * 4),
                   _folds(case["log_k"] + case["log_blowup"], case["rounds"], "babybear",
                          max(case["limbs"], case["point_limbs"])))
        b, f = one[0] * case["count"], one[1] * case["count"]
    elif kind in ("basefold_open", "sp1_open"):
        field = "babybear" if kind == "basefold_open" else "koalabear"
        w = case["width"] + case.get("width2", 0)
        s, log_n = 1 << case["log_k"], case["log_k"] + case["log_blowup"]
        # columns (and, for Basefold, codewords) read once, the batched MLE and
        # its halvings, the fold layers, the expected proof-of-work search
        b, f = _sum((4 * w * s, w * s * 16),
                    (4 * w << log_n, (w << log_n) * 16) if kind == "basefold_open"
                    else _lde(4, case["log_k"], case["log_blowup"]),
                    (16 * 4 * s, 2 * s * 2 * 64), _folds(log_n, case["log_k"], field, 4),
                    (0, (1 << case.get("pow_bits", 0)) * _PERM[field]))
    elif kind == "kary_fold":
        b = f = 0
        for r in range(case["rounds"]):
            n = 1 << (case["log_n"] - r * case["log_arity"])
            m = n >> case["log_arity"]
            b, f = _sum((b, f), _tree(m, -(-(1 << case["log_arity"]) // 8), "koalabear"),
                        (4 * (n + m), n * 8))
    elif kind == "strided_commit":
        h = 1 << case["log_h"]
        s = h // case["rows_per_query"]
        b = 4 * h * case["width"] + 32 * (2 * s - 1)
        f = _PERM["babybear"] * (h * -(-case["width"] // 8) + h - 1)
    else:
        inv = (0, (case["width"] << case["log_k"]) * case["log_k"] // 2 * 8)
        b, f = _sum(inv, _lde(case["width"], case["log_k"], case["log_blowup"]))
    return {"bytes": b, "flops": f}


# -------------------------------------------------------------- exact ----
def _dft(x, root, p):
    """out[j] = sum_i x[i] root^(ij) over the last axis, in 64-bit integers."""
    n = x.shape[-1]
    log_n = n.bit_length() - 1
    idx = torch.arange(n, device=x.device)
    rev = torch.zeros_like(idx)
    for b in range(log_n):
        rev |= ((idx >> b) & 1) << (log_n - 1 - b)
    x = x[..., rev]
    for b in range(log_n):
        half = 1 << b
        w = torch.ones(1, dtype=torch.int64, device=x.device)
        step = pow(root, n >> (b + 1), p)
        while w.numel() < half:  # powers of the stage's root, by doubling
            w = torch.cat([w, w * pow(step, w.numel(), p) % p])
        y = x.reshape(*x.shape[:-1], n // (2 * half), 2, half)
        u, v = y[..., 0, :], y[..., 1, :] * w % p
        x = torch.stack([(u + v) % p, (u - v) % p], dim=-2).reshape(*x.shape[:-1], n)
    return x


def exact(case, seed):
    if case["kind"] != "extend":
        return None
    s = prepare(case, seed)
    p, g = FIELDS[case["field"]].p, FIELDS[case["field"]].generator
    k, n = 1 << case["log_k"], 1 << (case["log_k"] + case["log_blowup"])
    x = s["x"].to(torch.int64)
    coeffs = _dft(x, pow(pow(g, (p - 1) // k, p), p - 2, p), p) * pow(k, p - 2, p) % p
    shift = torch.ones(1, dtype=torch.int64, device=x.device)
    while shift.numel() < k:  # powers of the coset shift, by doubling
        shift = torch.cat([shift, shift * pow(g, shift.numel(), p) % p])
    padded = torch.zeros(*x.shape[:-1], n, dtype=torch.int64, device=x.device)
    padded[..., :k] = coeffs * shift % p
    return _dft(padded, pow(g, (p - 1) // n, p), p).to(torch.int32)

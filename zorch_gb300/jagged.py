"""SP1's stacked BaseFold open on the GPU (drop-in for
zorch/pcs/jagged/open.py): the commit of a stacked region, the commit-and-fold
rounds, and the whole open with its interleaved sumcheck.

Each round's layer is a bit-reversed EF4 codeword [n, 4]; it is committed as
its [n/2, 8] base-limb rows (the adjacent conjugate pair of a fold is one row)
through the SP1 single-matrix commitment, whose separator-bound root the
transcript observes, and folded by BitReversedReedSolomon.fold. Round r+1's
commit runs in the same kernel as round r's fold (zc_fri_fold_commit_bitrev),
and every root is bound on the device, so the loop never synchronises with
the host. `StackedFoldCommit.run` takes each round's beta from the caller (the
reference's byte-match replays them the same way,
zorch/pcs/jagged/testing/open_test.py:90-128); `stacked_basefold_open` derives
them from the transcript after the round's sumcheck message (:266-290).
"""

from __future__ import annotations

from dataclasses import dataclass
from typing import Callable, Sequence

import numpy as np
import torch

from . import _lib
from .coding import BitReversedReedSolomon
from .commit import DigestLayers, SingleMatrixCommitmentScheme, leaves_layout
from .field import from_mont, full_u32, ptr, stream_handle, to_host
from .pcs import check_specs, layer_spec, open_layers, run_fold_rounds
from .transcript import DuplexTranscript


@dataclass
class StackedFoldLayer:
    """One committed fold layer: the codeword [n, 4], its digest layers over
    the [n/2, 8] pair rows, and the raw and separator-bound roots."""

    codeword: torch.Tensor
    digest_layers: DigestLayers
    raw_root: torch.Tensor
    bound_root: torch.Tensor

    @property
    def leaves(self) -> torch.Tensor:
        """The committed [n/2, 8] rows, a view of the codeword."""
        return self.codeword.reshape(self.codeword.shape[0] // 2, 8)


def sample_query_positions(t: DuplexTranscript, block_len: int, num_queries: int):
    """SP1's sample_bits rule (zorch/pcs/jagged/open.py:116-125): one squeeze
    per query, the CANONICAL value masked to log2(block_len) low bits."""
    if block_len <= 0 or block_len & (block_len - 1):
        raise ValueError(f"block_len must be a power of two, got {block_len}")
    t2, raw = t.sample(num_queries)
    canon = from_mont(t.field, raw)
    return t2, canon & (block_len - 1)


class StackedFoldCommit:
    """Commit -> bind -> fold rounds over a bit-reversed EF4 codeword."""

    def __init__(self, smcs: SingleMatrixCommitmentScheme, code: BitReversedReedSolomon) -> None:
        self.smcs = smcs
        self.code = code

    def commit_layer(self, cw: torch.Tensor) -> StackedFoldLayer:
        """smcs.commit(bitcast(cw).reshape(n/2, 8)) (zorch/pcs/jagged/open.py:278-282)."""
        n = cw.shape[0]
        if cw.dim() != 2 or cw.shape[1] != 4 or n < 2:
            raise ValueError("a stacked fold layer is an EF4 codeword [n >= 2, 4]")
        rows = cw.contiguous()
        bound, layers = self.smcs.commit_layout(leaves_layout(rows, n // 2, 1, 8, 0), 8)
        return StackedFoldLayer(rows, layers, layers.root, bound)

    def fold_commit(self, cw: torch.Tensor, beta: torch.Tensor,
                    level: int) -> tuple[torch.Tensor, StackedFoldLayer | None]:
        """Fold layer `cw` by `beta`; when the folded layer has >= 2 elements its
        commit runs fused with the fold (n >= 4)."""
        n = cw.shape[0]
        out = torch.empty((n // 2, 4), dtype=torch.int32, device=cw.device)
        if n < 4:
            return self.code.fold(cw, beta, out), None
        L = n // 4
        flat = torch.empty((2 * L - 1, 8), dtype=torch.int32, device=cw.device)
        _lib.check(_lib.lib().zc_fri_fold_commit_bitrev(
            self.smcs.perm.handle, ptr(cw), n, 1, ptr(beta.contiguous()), int(beta.numel() == 4),
            self.code.level_shift_mont(level), 0, ptr(out), ptr(flat), stream_handle()),
            "fri_fold_commit_bitrev")
        layers = DigestLayers(flat, L)
        bound = self.smcs.bind_root(layers.root, (L).bit_length() - 1, 8)
        return out, StackedFoldLayer(out, layers, layers.root, bound)

    def run(self, codeword: torch.Tensor, num_rounds: int,
            next_beta: Callable[[int, StackedFoldLayer], torch.Tensor]
            ) -> tuple[list[StackedFoldLayer], torch.Tensor]:
        """`num_rounds` commit-and-fold rounds; `next_beta(r, layer)` returns round
        r's EF4 beta (4 device words) after the layer is committed -- e.g. an
        observe of the bound root and a 4-squeeze challenge, or a replay.
        Returns the committed layers and the final folded codeword."""
        if num_rounds < 0 or (1 << num_rounds) > codeword.shape[0]:
            raise ValueError("more fold rounds than the codeword has halvings")
        cw = codeword
        layers: list[StackedFoldLayer] = []
        pending = None
        for r in range(num_rounds):
            layer = pending if pending is not None else self.commit_layer(cw)
            layers.append(layer)
            beta = next_beta(r, layer)
            cw, pending = self.fold_commit(cw, beta, self.code.level_of(cw.shape[0]))
        return layers, cw

    def run_replay(self, codeword: torch.Tensor, betas: Sequence[torch.Tensor] | torch.Tensor):
        """run() with the betas given up front ([R, 4] device words)."""
        return self.run(codeword, len(betas), lambda r, _layer: betas[r])

    def open_layers(self, layers: Sequence[StackedFoldLayer], positions: torch.Tensor,
                    check: bool = True):
        """Each layer's pair row opened at the halved positions a_i = q >> (i+1)
        (BitReversedReedSolomon.layer_positions; zorch/pcs/jagged/open.py:313-317):
        a list of (rows [Q, 8], proofs [depth_i, Q, 8]). `check=False` skips the
        range read-back for positions drawn below n (then a_i < n / 2^(i+1))."""
        idx = self.code.layer_positions(positions.to(torch.int32), len(layers))
        return [self.smcs.open_batch(i, layer.leaves, layer.digest_layers, check=check)
                for i, layer in zip(idx, layers)]


# ------------------------------------------------------------ stacked open --
@dataclass
class StackedRound:
    """One committed region (zorch/pcs/jagged/open.py:64-82): the [K, S]
    message block (Montgomery words), its bit-reversed codeword [K, n], the
    digest layers of its column-major SMCS commit and the bound commitment."""

    block: torch.Tensor
    codeword: torch.Tensor
    digest_layers: DigestLayers
    commitment: torch.Tensor


def stacked_commit(smcs: SingleMatrixCommitmentScheme, code: BitReversedReedSolomon,
                   block: torch.Tensor) -> StackedRound:
    """Encode the [K, S] block bit-reversed and commit its codeword columns
    (a leaf is a codeword position across the K columns)."""
    cw = code.encode(block)
    commitment, layers = smcs.commit(cw, column_major=True)
    return StackedRound(block, cw, layers, commitment)


@dataclass
class StackedOpenProof:
    """zorch/pcs/jagged/open.py:128-176: per round the bound component
    commitment, the fold layers' raw and bound roots, the sumcheck messages
    (s(0), s(1)), the final poly (codeword[0]), the proof-of-work witness, the
    per-round column evaluations, and the component and fold-layer openings
    (rows, sibling paths)."""

    component_commitments: list
    fri_raw_roots: torch.Tensor       # [v, 8]
    fri_commitments: torch.Tensor     # [v, 8]
    univariate_messages: torch.Tensor  # [v, 2, 4]
    final_poly: torch.Tensor          # [4]
    pow_witness: torch.Tensor         # [1]
    batch_evals: list                 # per round [K, 4]
    component_openings: list          # per round (rows [Q, K], paths [depth, Q, 8])
    query_openings: list              # per layer (rows [Q, 8], paths [depth_i, Q, 8])
    positions: torch.Tensor           # [Q]


def _ef4_encode(code: BitReversedReedSolomon, mle: torch.Tensor) -> torch.Tensor:
    """Bit-reversed encode of an EF4 message [S, 4] limb by limb (the base-field
    roots act on each coefficient) -> [n, 4]."""
    L, st = _lib.lib(), stream_handle()
    S = mle.shape[0]
    limbs = torch.empty((4, S), dtype=torch.int32, device=mle.device)
    _lib.check(L.zc_ef4_limbs(ptr(mle), S, 1, ptr(limbs), st), "ef4_limbs")
    cw = code.encode(limbs)
    out = torch.empty((cw.shape[1], 4), dtype=torch.int32, device=mle.device)
    _lib.check(L.zc_ef4_limbs(ptr(cw), cw.shape[1], 0, ptr(out), st), "ef4_limbs")
    return out


def stacked_basefold_open(smcs: SingleMatrixCommitmentScheme, code: BitReversedReedSolomon,
                          rounds, z_final: torch.Tensor, dense_eval: torch.Tensor,
                          log_stacking_height: int, *, num_queries: int, pow_bits: int,
                          transcript: DuplexTranscript):
    """The stacked BaseFold open (zorch/pcs/jagged/open.py:362-460: prologue
    :185-229, fold zone :237-330, component queries :333-359) on the GPU:
    evaluate every round's columns at the stacking point, observe dense_eval and
    the evaluations, batch the rounds with partial-Lagrange weights over
    ceil(log2 total width) EF4 challenges, re-encode the batched MLE, observe the
    round count, then per round: sumcheck message, SMCS commit of the
    pre-fold [n/2, 8] rows, observe message and bound root, EF4 beta, fold the
    codeword, MLE and claim; observe the final poly, grind, draw SP1 query
    positions and open every fold layer and every committed round."""
    if not rounds:
        raise ValueError("the stacked open needs at least one committed round")
    if log_stacking_height < 1:
        raise ValueError(f"need at least one stacking variable, got "
                         f"log_stacking_height={log_stacking_height}")
    if z_final.shape[0] < log_stacking_height:
        raise ValueError(f"z_final has {z_final.shape[0]} coordinates, fewer than "
                         f"log_stacking_height={log_stacking_height}")
    S = 1 << log_stacking_height
    if code.message_len != S:
        raise ValueError(f"code message_len {code.message_len} != stacking height {S}")
    if any(rd.block.shape[1] != S for rd in rounds):
        raise ValueError(f"every round block must stack to height {S}")
    f, L, st = code.field, _lib.lib(), stream_handle()
    dev = z_final.device
    v = log_stacking_height
    n = code.block_len
    zs = z_final[-v:].contiguous()
    t = transcript._copy()
    # prologue: per-round evaluations at the stacking point
    batch_evals = []
    for rd in rounds:
        K = rd.block.shape[0]
        out = torch.empty((K, 4), dtype=torch.int32, device=dev)
        nb = L.zc_eval_mle_workspace_bytes(K, v)
        ws = torch.empty((nb + 15) // 4, dtype=torch.int32, device=dev)
        _lib.check(L.zc_eval_mle(f.id, ptr(rd.block.contiguous()), K, v, ptr(zs), ptr(out),
                                 ptr(ws), nb, st), "eval_mle")
        batch_evals.append(out)
    t.observe_(dense_eval.reshape(-1))
    for e in batch_evals:
        t.observe_(e.reshape(-1))
    total = sum(int(rd.block.shape[0]) for rd in rounds)
    nbv = (total - 1).bit_length() if total > 1 else 0
    chal = t.sample_(4 * nbv) if nbv else torch.empty(4, dtype=torch.int32, device=dev)
    mle = torch.empty((S, 4), dtype=torch.int32, device=dev)
    claim = torch.empty(4, dtype=torch.int32, device=dev)
    off = 0
    for rd, e in zip(rounds, batch_evals):
        K = rd.block.shape[0]
        acc = int(off > 0)
        _lib.check(L.zc_rlc_columns_ex(f.id, ptr(rd.block.contiguous()), S, K, ptr(chal), nbv,
                                       off, acc, ptr(mle), st), "rlc mle")
        _lib.check(L.zc_rlc_values(f.id, ptr(e), K, ptr(chal), nbv, off, acc, ptr(claim), st),
                   "rlc values")
        off += K
    # fold zone
    cw = _ef4_encode(code, mle)
    t.observe_(full_u32(1, f.mont(v), dev))  # a fill kernel: no host copy
    zinv = torch.empty_like(zs)  # 1/z per stacking coordinate, on the device
    _lib.check(L.zc_ef4_inv(f.id, ptr(zs), ptr(zinv), v, st), "ef4_inv")
    eq = torch.empty((max(S // 2, 1), 4), dtype=torch.int32, device=dev)
    nb = L.zc_eq_expand_workspace_bytes(v - 1)
    ews = torch.empty(max((nb + 15) // 4, 4), dtype=torch.int32, device=dev)
    _lib.check(L.zc_eq_expand(f.id, ptr(zs), v - 1, ptr(eq), ptr(ews), nb, st), "eq_expand")
    fr = run_fold_rounds(smcs.perm, code, cw, v, 4, t, bind=True,
                         sumcheck=(mle, eq, claim, zinv))
    cw = fr.final_layer
    final_poly = cw[0].contiguous()
    t.observe_(final_poly)
    t, witness = t.grind(pow_bits)  # the query-phase proof of work (:304-307)
    witness = witness.reshape(1)
    t, positions = sample_query_positions(t, n, num_queries)
    positions = positions.to(torch.int32)
    # the rounds' matrices, then every fold layer at a_i = q >> (i+1)
    # (BitReversedReedSolomon.layer_positions); positions are masked below n
    specs = []
    for rd in rounds:
        K = rd.codeword.shape[0]
        specs.append((leaves_layout(rd.codeword, n, K, 1, n), rd.digest_layers, K, 0))
    check_specs(specs)
    opened = [(op.row, op.path) for op in
              open_layers(specs + [layer_spec(ly, i, True) for i, ly in enumerate(fr.layers)],
                          positions, check=False)]
    proof = StackedOpenProof(
        [rd.commitment for rd in rounds], fr.raw_roots, fr.roots, fr.msgs.view(v, 2, 4),
        final_poly, witness, batch_evals, opened[:len(specs)], opened[len(specs):], positions)
    return proof, t


def _ef_eval_mle_msb(f, values: list, point: list) -> tuple:
    """MLE of `values` (EF4 tuples, 2^m of them) at `point` (m EF4 tuples),
    point[0] binding the most significant index bit -- the eq-table order of
    eval_mle (zorch/poly/eq.py:55-62)."""
    cur = list(values)
    for z in point:
        half = len(cur) // 2
        cur = [f.ef_add(cur[i], f.ef_mul(z, f.ef_sub(cur[half + i], cur[i]))) for i in range(half)]
    return cur[0]


def stacked_basefold_verify(smcs: SingleMatrixCommitmentScheme, code: BitReversedReedSolomon,
                            round_widths: Sequence[int], z_final, dense_eval,
                            log_stacking_height: int, proof: StackedOpenProof, transcript,
                            *, num_queries: int, pow_bits: int):
    """Verify a stacked BaseFold open on the host (stacked_basefold_verify,
    zorch/pcs/jagged/verifier.py:165-356); returns (transcript, ok).

    `transcript` is a HostDuplexTranscript at the state the prover's open
    started from. Checks, in the open's absorb order: SP1's stacking identity
    (dense_eval = the MLE of the concatenated batch evaluations at the leading
    coordinates), the staggered batching, every interleaved sumcheck round
    against the running claim, each bound fold root against its raw root, the
    proof of work, the query positions, every component and fold-layer
    opening against its commitment, the batched component rows against fold
    layer 0, and the bit-reversed fold chain down to the final poly. Malformed
    shapes raise ValueError, as the reference does; a wrong proof gives False."""
    f = code.field
    host = lambda x: to_host(x) if torch.is_tensor(x) else np.asarray(x, np.uint32)  # noqa: E731
    ef = lambda w: f.ef_from_mont([int(v) for v in w])  # noqa: E731
    v = log_stacking_height
    n = code.block_len
    if v < 1:
        raise ValueError(f"need at least one stacking variable, got "
                         f"log_stacking_height={log_stacking_height}")
    if num_queries < 1:
        raise ValueError(f"need at least one query, got num_queries={num_queries}")
    if not (len(proof.component_commitments) == len(round_widths) == len(proof.batch_evals)
            == len(proof.component_openings)):
        raise ValueError(f"round mismatch: {len(proof.component_commitments)} component "
                         f"commitments, {len(round_widths)} widths, "
                         f"{len(proof.batch_evals)} batch evals, "
                         f"{len(proof.component_openings)} component openings")
    evals = [host(e).reshape(-1, 4) for e in proof.batch_evals]
    for r, (e, k) in enumerate(zip(evals, round_widths)):
        if e.shape[0] != k:
            raise ValueError(f"round {r} batch evals must cover its {k} stacked columns, "
                             f"got {e.shape[0]}")
    msgs = host(proof.univariate_messages).reshape(-1, 8)
    raw = host(proof.fri_raw_roots).reshape(-1, 8)
    bound = host(proof.fri_commitments).reshape(-1, 8)
    if msgs.shape[0] != v:
        raise ValueError(f"need one (s(0), s(1)) message per stacking variable ({v}), "
                         f"got {msgs.shape[0]}")
    if bound.shape[0] != v or raw.shape[0] != v or len(proof.query_openings) != v:
        raise ValueError(f"need one committed fold layer per stacking variable ({v})")
    zf = [ef(r) for r in host(z_final).reshape(-1, 4)]
    if len(zf) < v:
        raise ValueError(f"the folded point must carry at least the {v} stacking "
                         f"variables, got {len(zf)}")
    stack_point, batch_point = zf[len(zf) - v:], zf[:len(zf) - v]
    flat = [ef(r) for e in evals for r in e]
    width = 1 << len(batch_point)
    if len(flat) > width:
        raise ValueError(f"{len(flat)} stacked columns do not fit the {len(batch_point)} "
                         f"leading point variables")
    de = host(dense_eval).reshape(-1)
    ok = ef(de) == _ef_eval_mle_msb(f, flat + [(0, 0, 0, 0)] * (width - len(flat)),
                                    batch_point)
    t = transcript.observe(de)
    for e in evals:
        t = t.observe(e.reshape(-1))
    total = sum(int(k) for k in round_widths)
    nbv = (total - 1).bit_length() if total > 1 else 0
    chal = []
    if nbv:
        t, s = t.sample(4 * nbv)
        chal = [ef(s[4 * j:4 * j + 4]) for j in range(nbv)]

    def weight(idx: int) -> tuple:
        w = (1, 0, 0, 0)
        for j, r in enumerate(chal):
            bit = (idx >> (nbv - 1 - j)) & 1
            w = f.ef_mul(w, r if bit else f.ef_sub((1, 0, 0, 0), r))
        return w

    wts = [weight(c) for c in range(total)]
    claim = (0, 0, 0, 0)
    for c, x in enumerate(flat):
        claim = f.ef_add(claim, f.ef_mul(wts[c], x))
    t = t.observe([f.mont(v)])
    betas = []
    for i in range(v):
        s0, s1 = ef(msgs[i, :4]), ef(msgs[i, 4:])
        x = stack_point[v - 1 - i]
        ok &= claim == f.ef_add(f.ef_mul(f.ef_sub((1, 0, 0, 0), x), s0), f.ef_mul(x, s1))
        t = t.observe(msgs[i])
        t, b = t.observe_and_sample(bound[i], 4)
        beta = ef(b)
        betas.append(beta)
        claim = f.ef_add(s0, f.ef_mul(beta, s1))
        log_h = (n >> (i + 1)).bit_length() - 1
        ok &= np.array_equal(smcs.bind_root_host(raw[i], log_h, 8), bound[i])
    final = host(proof.final_poly).reshape(-1)
    t = t.observe(final)
    t, ok_pow = t.check_witness(host(proof.pow_witness).reshape(-1), pow_bits=pow_bits)
    ok &= bool(ok_pow)
    t, sq = t.sample(num_queries)
    positions = [f.canon(int(x)) & (n - 1) for x in sq]
    if [int(x) for x in host(proof.positions).reshape(-1)] != positions:
        return t, False
    # Merkle phase
    from .commit import VerifyCode

    for r, (rows, paths) in enumerate(proof.component_openings):
        rows, paths = host(rows), host(paths)
        for qi, q in enumerate(positions):
            ok &= smcs.verify_batch(proof.component_commitments[r], (n, int(round_widths[r])),
                                    q, rows[qi], paths[:, qi]) == VerifyCode.OK
    for i, (rows, paths) in enumerate(proof.query_openings):
        rows, paths = host(rows), host(paths)
        for qi, q in enumerate(positions):
            ok &= smcs.verify_batch(bound[i], (n >> (i + 1), 8), q >> (i + 1), rows[qi],
                                    paths[:, qi]) == VerifyCode.OK
    if not ok:
        return t, False
    # fold consistency: batched component rows at q == fold layer 0's leg; then
    # each opened pair (f(x), f(-x)) folds to the next layer's value
    shift = code.coset_shift or 1
    inv2 = pow(2, f.p - 2, f.p)
    comp_rows = [host(rows) for rows, _ in proof.component_openings]
    layer_rows = [host(rows).reshape(-1, 2, 4) for rows, _ in proof.query_openings]
    final_ef = ef(final)
    for qi, q in enumerate(positions):
        comp, off = (0, 0, 0, 0), 0
        for rows in comp_rows:
            for c, xw in enumerate(rows[qi]):
                comp = f.ef_add(comp, f.ef_scale(wts[off + c], f.canon(int(xw))))
            off += rows.shape[1]
        ok &= comp == ef(layer_rows[0][qi][q & 1])
        for i in range(v):
            ni = n >> i
            m = ni.bit_length() - 1
            a = q >> (i + 1)
            e = int(bin(a)[2:].zfill(m - 1)[::-1], 2) if m > 1 else 0  # brev_{m-1}(a)
            xpt = pow(shift, 1 << i, f.p) * pow(f.root_of_unity(m), e, f.p) % f.p
            lo, hi = ef(layer_rows[i][qi][0]), ef(layer_rows[i][qi][1])
            folded = f.ef_add(f.ef_scale(f.ef_add(lo, hi), inv2),
                              f.ef_scale(f.ef_mul(betas[i], f.ef_sub(lo, hi)),
                                         pow(2 * xpt % f.p, f.p - 2, f.p)))
            want = ef(layer_rows[i + 1][qi][a & 1]) if i + 1 < v else final_ef
            ok &= folded == want
    return t, bool(ok)


class GraphedStackedOpen:
    """stacked_basefold_open over fixed committed rounds captured once into a
    CUDA graph: the batch evaluations, the batching, every interleaved
    sumcheck round with its fused fold-and-commit, the grind, the SP1 query
    positions and all openings replay with one launch. `replay(z_final,
    dense_eval, transcript)` copies the statement and the transcript state
    into static inputs and returns (proof, transcript) -- static tensors the
    next replay overwrites. The rounds' device buffers are baked into the
    graph."""

    def __init__(self, smcs: SingleMatrixCommitmentScheme, code: BitReversedReedSolomon,
                 rounds: Sequence[StackedRound], num_vars: int, log_stacking_height: int, *,
                 num_queries: int, pow_bits: int, device="cuda") -> None:
        self.args = (smcs, code, list(rounds))
        self.log_s = log_stacking_height
        self.kw = dict(num_queries=num_queries, pow_bits=pow_bits)
        self.z = torch.zeros((num_vars, 4), dtype=torch.int32, device=device)
        self.dense = torch.zeros(4, dtype=torch.int32, device=device)
        self.state = torch.zeros(_lib.DUPLEX_WORDS, dtype=torch.int32, device=device)
        self._run()  # kernel attributes, allocator warm-up
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self.out = self._run()

    def _run(self):
        smcs, code, rounds = self.args
        t = DuplexTranscript(smcs.perm, self.state)
        return stacked_basefold_open(smcs, code, rounds, self.z, self.dense, self.log_s,
                                     transcript=t, **self.kw)

    def replay(self, z_final: torch.Tensor, dense_eval: torch.Tensor,
               transcript: DuplexTranscript):
        if z_final.shape != self.z.shape:
            raise ValueError(f"point shape {tuple(z_final.shape)} != captured "
                             f"{tuple(self.z.shape)}")
        self.z.copy_(z_final, non_blocking=True)
        self.dense.copy_(dense_eval.reshape(-1), non_blocking=True)
        self.state.copy_(transcript.state, non_blocking=True)
        self.graph.replay()
        return self.out

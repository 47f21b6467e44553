"""The one-call fold rounds (zc_fold_rounds behind the FRI, Basefold and SP1
opens) against the same rounds run one step at a time through the public
classes and entries, at the edges of its shapes: one round, as many rounds as
the codeword halves, base and EF4 layers and challenges, both codeword orders,
a first layer that is committed already, bound roots, and the interleaved
sumcheck from one variable up past one CTA's and one grid's worth of pairs.
The batched opening likewise against the single one. Words are equal exactly."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from zorch_gb300 import _lib  # noqa: E402
from zorch_gb300.coding import BitReversedReedSolomon, ReedSolomon  # noqa: E402
from zorch_gb300.commit import (MerkleTree, Poseidon2, SingleMatrixCommitmentScheme,  # noqa: E402
                                koalabear16_params)
from zorch_gb300.field import BABYBEAR, KOALABEAR, ptr, stream_handle, to_device  # noqa: E402
from zorch_gb300.jagged import StackedFoldCommit  # noqa: E402
from zorch_gb300.pcs import (FoldState, PreFoldPairCommitRound, fold_rounds, layer_spec,  # noqa: E402
                             open_layer, open_layers, run_fold_rounds)
from zorch_gb300.transcript import DuplexTranscript  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    _lib.check(_lib.lib().zc_init(0), "init")


def _words(field, *shape, seed=1):
    x = np.random.default_rng(seed).integers(0, field.p, size=shape, dtype=np.uint64)
    return to_device(x.astype(np.uint32)).reshape(shape)


def _eq(a, b):
    assert a.shape == b.shape and torch.equal(a, b)


@pytest.mark.parametrize("br", [False, True])
@pytest.mark.parametrize("limbs", [1, 4])
@pytest.mark.parametrize("ef", [False, True])
@pytest.mark.parametrize("log_n,rounds", [(1, 1), (2, 1), (2, 2), (3, 2), (7, 7), (10, 4), (16, 3)])
def test_rounds_equal_single_steps(br, limbs, ef, log_n, rounds):
    perm = Poseidon2.builtin(BABYBEAR)
    n = 1 << log_n
    code = (BitReversedReedSolomon(n // 2, 2, BABYBEAR) if br else
            ReedSolomon(n // 2, 2, BABYBEAR, coset_shift=31, generator=31))
    cw = _words(BABYBEAR, n, 4) if ef else _words(BABYBEAR, n)
    tree = MerkleTree(perm)
    rnd = PreFoldPairCommitRound(code, tree, limbs, last_round=rounds - 1)
    t0 = DuplexTranscript.new(perm).observe(_words(BABYBEAR, 5, seed=2))
    st, t1, roots = fold_rounds(rnd, FoldState(cw), t0, rounds)
    for first in (None, rnd.commit_layer(cw)):
        t = t0._copy()
        got = run_fold_rounds(perm, code, cw, rounds, limbs, t, first)
        _eq(got.final_layer, st.codeword)
        _eq(got.roots, torch.stack(list(roots)))
        _eq(got.betas, torch.stack(list(st.betas)))
        _eq(t.state, t1.state)
        assert len(got.layers) == rounds
        for a, b in zip(got.layers, st.layers):
            _eq(a.codeword, b.codeword)
            _eq(a.digest_layers.flat, b.digest_layers.flat)
        pos = torch.tensor([0, n - 1, n // 2, n // 3], dtype=torch.int32, device="cuda")
        specs = [layer_spec(ly, i, br) for i, ly in enumerate(got.layers)]
        if got.layers[-1].digest_layers.depth == 0:  # one leaf, no path: both refuse it
            with pytest.raises(_lib.ZcError):
                open_layers(specs, pos)
            with pytest.raises(_lib.ZcError):
                open_layer(tree, got.layers[-1], pos, rounds - 1, br)
            specs.pop()
        for i, (layer, op) in enumerate(zip(got.layers, open_layers(specs, pos))):
            want = open_layer(tree, layer, pos, i, br)
            _eq(op.row, want.row)
            _eq(op.path, want.path)


@pytest.mark.parametrize("v", [1, 2, 3, 9, 11, 18])
@pytest.mark.parametrize("sp1", [False, True])
def test_rounds_with_sumcheck(orc, v, sp1):
    field = KOALABEAR if sp1 else BABYBEAR
    perm = koalabear16_params(orc.load_sp1_fixture()) if sp1 else Poseidon2.builtin(BABYBEAR)
    n, limbs, L, st = 2 << v, 4 if sp1 else 1, _lib.lib(), stream_handle()
    code = (BitReversedReedSolomon(1 << v, 2, field) if sp1 else
            ReedSolomon(1 << v, 2, field, coset_shift=31))
    cw = _words(field, n, 4, seed=3)
    mle, eq = _words(field, 1 << v, 4, seed=4), _words(field, 1 << (v - 1), 4, seed=5)
    zinv, claim0 = _words(field, v, 4, seed=6), _words(field, 4, seed=7)
    # one step at a time
    t = DuplexTranscript.new(perm)
    claim, m, e, cur, pending = claim0.clone(), mle, eq, cw, None
    msgs = torch.empty((v, 8), dtype=torch.int32, device="cuda")
    ws = torch.empty(L.zc_sumcheck_workspace_bytes() // 4, dtype=torch.int32, device="cuda")
    fold = StackedFoldCommit(SingleMatrixCommitmentScheme(perm), code) if sp1 else None
    rnd = PreFoldPairCommitRound(code, MerkleTree(perm), limbs)
    roots, raws, betas = [], [], []
    for i in range(v):
        M = 1 << (v - 1 - i)
        _lib.check(L.zc_sumcheck_message(field.id, ptr(m), M, ptr(e), ptr(claim),
                                         ptr(zinv[v - 1 - i]), ptr(msgs[i]), ptr(ws),
                                         ws.numel() * 4, st))
        layer = pending if pending is not None else (fold.commit_layer(cur) if sp1
                                                     else rnd.commit_layer(cur))
        t.observe_(msgs[i])
        root = layer.bound_root if sp1 else layer.root
        beta = t.observe_and_sample_(root, limbs)
        roots.append(root)
        raws.append(layer.raw_root if sp1 else layer.root)
        betas.append(beta)
        if sp1:
            nxt, pending = fold.fold_commit(cur, beta, code.level_of(cur.shape[0]))
        elif i < v - 1:
            nxt, pending = rnd.fold_commit(cur, beta, i)
        else:
            nxt, pending = code.fold(cur, beta), None
        m2 = torch.empty((M, 4), dtype=torch.int32, device="cuda")
        e2 = torch.empty((M // 2, 4), dtype=torch.int32, device="cuda") if M >= 2 else None
        _lib.check(L.zc_sumcheck_fold(field.id, ptr(m), M, ptr(beta), limbs, ptr(msgs[i]), ptr(m2),
                                      ptr(e) if M >= 2 else None, ptr(e2), ptr(claim), st))
        m, e, cur = m2, e2, nxt
    # one call
    t1, claim1 = DuplexTranscript.new(perm), claim0.clone()
    got = run_fold_rounds(perm, code, cw, v, limbs, t1, bind=sp1,
                          sumcheck=(mle, eq, claim1, zinv))
    _eq(got.msgs, msgs)
    _eq(got.roots, torch.stack(roots))
    if sp1:
        _eq(got.raw_roots, torch.stack(raws))
    _eq(got.betas, torch.stack(betas))
    _eq(got.final_layer, cur)
    _eq(claim1, claim)
    _eq(t1.state, t.state)


def test_rounds_refuse_bad_shapes():
    import ctypes

    L, perm = _lib.lib(), Poseidon2.builtin(BABYBEAR)
    d = _lib.FoldRoundsDesc()
    assert L.zc_fold_rounds(perm.handle, ctypes.byref(d), stream_handle()) == 7  # no rounds
    d.rounds, d.log_n = 3, 2
    assert L.zc_fold_rounds(perm.handle, ctypes.byref(d), stream_handle()) == 7

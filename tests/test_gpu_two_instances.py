"""Opens whose transcript runs another Poseidon2 instance than the tree: every
challenge comes from the transcript's permutation and every digest from the
tree's. The rounds equal the same rounds run one step at a time, the host
verifiers over a transcript of that instance accept the proofs, and an instance
of equal constants behind another handle changes no word."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from zorch_gb300 import _lib  # noqa: E402
from zorch_gb300.coding import BitReversedReedSolomon, ReedSolomon  # noqa: E402
from zorch_gb300.commit import (MerkleTree, Poseidon2, SingleMatrixCommitmentScheme,  # noqa: E402
                                koalabear16_params)
from zorch_gb300.field import BABYBEAR, KOALABEAR, to_device, to_host  # noqa: E402
from zorch_gb300.pcs import (BasefoldProver, BasefoldVerifier, FoldState, FriParams,  # noqa: E402
                             FriProver, FriVerifier, PreFoldPairCommitRound, fold_rounds)
from zorch_gb300.stage import OpeningClaim, OpeningWitness  # noqa: E402
from zorch_gb300.transcript import DuplexTranscript, HostDuplexTranscript  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    _lib.check(_lib.lib().zc_init(0), "init")


def _words(field, *shape, seed=1):
    x = np.random.default_rng(seed).integers(0, field.p, size=shape, dtype=np.uint64)
    return to_device(x.astype(np.uint32)).reshape(shape)


def _babybear(orc, change: int) -> Poseidon2:
    """The built-in instance's constants as a run-time instance; `change` is
    added to the first round constant."""
    ei, et, ir, dg = orc.Poseidon2.babybear16().export_canonical()
    ei = ei.copy()
    ei[0, 0] = (int(ei[0, 0]) + change) % BABYBEAR.p
    return Poseidon2.from_params(BABYBEAR, 7, ei, et, ir, dg)


def _instances(orc, name):
    """(tree's instance, transcript's instance, whether they are equal)."""
    kb, sp1 = orc.load_koalabear_fixture(), orc.load_sp1_fixture()
    return {
        "builtin, run-time": lambda: (Poseidon2.builtin(), _babybear(orc, 1), False),
        "run-time, builtin": lambda: (_babybear(orc, 1), Poseidon2.builtin(), False),
        "builtin, the same constants": lambda: (Poseidon2.builtin(), _babybear(orc, 0), True),
        "koalabear, sp1": lambda: (koalabear16_params(kb), koalabear16_params(sp1), False),
        "koalabear twice": lambda: (koalabear16_params(kb), koalabear16_params(kb), True),
    }[name]()


PAIRS = ["builtin, run-time", "run-time, builtin", "builtin, the same constants",
         "koalabear, sp1", "koalabear twice"]


@pytest.mark.parametrize("fuse_hop", [False, True])
@pytest.mark.parametrize("limbs", [1, 2, 4])
@pytest.mark.parametrize("pair", PAIRS)
def test_commit_phase(orc, pair, limbs, fuse_hop):
    tree_p, t_p, _ = _instances(orc, pair)
    f = tree_p.field
    log_n, rounds = 11, 9
    code = ReedSolomon(1 << (log_n - 1), 2, f, coset_shift=f.generator)
    cw = _words(f, 1 << log_n)
    tree = MerkleTree(tree_p)
    t0 = DuplexTranscript.new(t_p).observe(_words(f, 5, seed=2))
    # every step by itself
    t, want, cur = t0._copy(), [], cw
    steps = PreFoldPairCommitRound(code, tree, limbs)
    for i in range(rounds):
        layer = steps.commit_layer(cur)
        beta = t.observe_and_sample_(layer.root, limbs)
        want.append((layer.root, beta))
        cur = code.fold(cur, beta)
    rnd = PreFoldPairCommitRound(code, tree, limbs, last_round=rounds - 1, fuse_hop=fuse_hop)
    st, t1, roots = fold_rounds(rnd, FoldState(cw), t0, rounds)
    assert torch.equal(t1.state, t.state)
    assert all(torch.equal(r, w) for r, (w, _) in zip(roots, want))
    proof, t2, _ = FriProver(FriParams(code, tree, rounds, 7, limbs)).commit_phase(cw, t0)
    assert torch.equal(proof.roots, torch.stack([w for w, _ in want]))
    assert all(torch.equal(b, w) for b, (_, w) in zip(proof.betas, want))
    assert torch.equal(proof.final_layer, cur)
    assert torch.equal(proof.positions, t.sample_positions_(1 << log_n, 7, values=cur))
    assert torch.equal(t2.state, t.state)


@pytest.mark.parametrize("pair", PAIRS)
def test_fri_prove(orc, pair):
    tree_p, t_p, same = _instances(orc, pair)
    f = tree_p.field
    code = ReedSolomon(1 << 8, 2, f, coset_shift=f.generator)
    params = FriParams(code, MerkleTree(tree_p), 8, 5, 4)
    prover = FriProver(params)
    polys = [_words(f, 1 << 8, seed=3), _words(f, 1 << 8, seed=4)]
    zs = [(5, 7, 11, 13), (9, 2, 0, 1)]
    roots, data = prover.commit(polys)
    res = prover.prove(OpeningClaim(roots, zs), OpeningWitness(data), DuplexTranscript.new(t_p))
    check = lambda p: FriVerifier(params).verify(OpeningClaim(roots, zs),  # noqa: E731
                                                 res.reduction_proof, HostDuplexTranscript(p)).ok
    assert check(t_p)
    assert check(tree_p) == same


@pytest.mark.parametrize("pair", PAIRS)
def test_basefold_open(orc, pair):
    tree_p, t_p, same = _instances(orc, pair)
    f, v = tree_p.field, 7
    code = ReedSolomon(1 << v, 2, f, coset_shift=f.generator)
    tree = MerkleTree(tree_p, column_major=True)
    prover = BasefoldProver(code, tree, num_queries=5)
    committed = [prover.commit_columns(_words(f, w, 1 << v, seed=10 + w)) for w in (3, 2)]
    roots, datas = [r for r, _ in committed], [d for _, d in committed]
    z = _words(f, v, 4, seed=20)
    values, proof, t = prover.open_batch(datas, z, DuplexTranscript.new(t_p))
    check = lambda p: BasefoldVerifier(code, tree, 5).verify_batch(  # noqa: E731
        roots, [z], values, proof, HostDuplexTranscript(p))
    ok, host = check(t_p)
    assert ok and np.array_equal(host.state, to_host(t.state))
    assert check(tree_p)[0] == same


@pytest.mark.parametrize("name", ["other", "equal"])
def test_stacked_open(orc, name):
    from zorch_gb300.jagged import (_ef_eval_mle_msb, stacked_basefold_open,
                                    stacked_basefold_verify, stacked_commit)

    f, v, widths = KOALABEAR, 6, (3, 2)
    sp1 = koalabear16_params(orc.load_sp1_fixture())
    t_p = koalabear16_params(orc.load_sp1_fixture() if name == "equal"
                             else orc.load_koalabear_fixture())
    code = BitReversedReedSolomon(1 << v, 2, f)
    smcs = SingleMatrixCommitmentScheme(sp1)
    rounds = [stacked_commit(smcs, code, _words(f, w, 1 << v, seed=30 + w)) for w in widths]
    z = _words(f, v + 3, 4, seed=40)
    open_ = lambda de: stacked_basefold_open(  # noqa: E731
        smcs, code, rounds, z, de, v, num_queries=5, pow_bits=3,
        transcript=DuplexTranscript.new(t_p))
    probe, _ = open_(_words(f, 4, seed=41))
    flat = [f.ef_from_mont(r) for e in probe.batch_evals for r in to_host(e).reshape(-1, 4)]
    de = np.array(f.ef_to_mont(_ef_eval_mle_msb(
        f, flat + [(0, 0, 0, 0)] * (8 - len(flat)),
        [f.ef_from_mont(r) for r in to_host(z)[:3]])), np.uint32)
    proof, _ = open_(to_device(de))
    check = lambda p: stacked_basefold_verify(  # noqa: E731
        smcs, code, list(widths), z, de, v, proof, HostDuplexTranscript(p), num_queries=5,
        pow_bits=3)[1]
    assert check(t_p)
    assert check(sp1) == (name == "equal")

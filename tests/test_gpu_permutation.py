"""Every form of the width-16 permutation on the GPU against the oracle: one
state per thread (zc_poseidon2_permute), the half-warp form (a transcript's
absorb chain) and the quarter- and half-warp forms of a tree's narrow levels,
for the instances with kernels of their own and for run-time instances whose
round counts and exponents sit at the edges of what zc_poseidon2_create takes.
Words at the ends of [0, p) are among the inputs: equality is exact."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from zorch_gb300 import _lib  # noqa: E402
from zorch_gb300.commit import MerkleTree, Poseidon2, koalabear16_params  # noqa: E402
from zorch_gb300.field import BABYBEAR, KOALABEAR, to_device, to_host  # noqa: E402
from zorch_gb300.transcript import DuplexTranscript  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    _lib.check(_lib.lib().zc_init(0), "init")


def _random_instance(orc, field, alpha, rfh, rp, j, seed):
    rng = np.random.default_rng(seed)
    p = (BABYBEAR if field == 0 else KOALABEAR).p
    draw = lambda *s: rng.integers(0, p, size=s, dtype=np.uint64).astype(np.uint32)  # noqa: E731
    ei, et, ir, dg = draw(rfh, 16), draw(rfh, 16), draw(rp), draw(16)
    dg[:4] = [0, 1, p - 1, p // 2]
    if rp:
        ir[0] = p - 1
    return (Poseidon2.from_params(field, alpha, ei, et, ir, dg, j),
            orc.Poseidon2.from_canonical(field, alpha, ei, et, ir, dg, j))


def _instance(orc, name):
    if name == "bb16":
        return Poseidon2.builtin(BABYBEAR), orc.Poseidon2.babybear16()
    if name == "kb16":
        return (koalabear16_params(orc.load_koalabear_fixture()),
                orc.Poseidon2.koalabear16_golden())
    if name == "sp1":
        return koalabear16_params(orc.load_sp1_fixture()), orc.sp1_koalabear16()
    if name[0] in ("plonky3", "sp1"):  # the two diagonals with other rounds and scales
        _, rp, j = name
        p, rng = KOALABEAR.p, np.random.default_rng(rp)
        h = lambda k: pow(2, -k, p)  # noqa: E731
        d = ([-2, 1, 2, h(1), 3, 4, -h(1), -3, -4, h(8), h(3), h(24), -h(8), -h(3), -h(4), -h(24)]
             if name[0] == "plonky3" else [-2] + [1 << i for i in range(14)] + [1 << 15])
        ei, et = (rng.integers(0, p, size=(4, 16), dtype=np.uint64).astype(np.uint32)
                  for _ in range(2))
        ir = rng.integers(0, p, size=rp, dtype=np.uint64).astype(np.uint32)
        dg = np.asarray([x * j % p for x in d], np.uint32)
        return (Poseidon2.from_params(1, 3, ei, et, ir, dg, j),
                orc.Poseidon2.from_canonical(1, 3, ei, et, ir, dg, j))
    field, alpha, rfh, rp, j = name
    return _random_instance(orc, field, alpha, rfh, rp, j, 7 * rp + alpha)


INSTANCES = ["bb16", "kb16", "sp1",
             # (field, alpha, half the full rounds, partial rounds, j)
             (0, 7, 4, 13, 1), (0, 7, 4, 13, 5), (0, 5, 3, 1, 1), (0, 3, 1, 2, 2013265920),
             (0, 11, 4, 14, 1), (1, 3, 4, 20, 1), (1, 3, 4, 20, 1057030144), (1, 3, 4, 12, 2),
             (1, 5, 8, 15, 1), (1, 7, 2, 16, 3), (1, 3, 4, 17, 1), (0, 7, 4, 26, 1),
             (1, 3, 1, 64, 9), (0, 7, 8, 29, 1),
             *[("plonky3", rp, j) for rp, j in [(1, 1), (2, 1), (3, 1), (20, 1), (33, 1), (20, 7)]],
             *[("sp1", rp, j) for rp, j in [(1, 5), (2, 1), (21, 1057030144), (64, 2130706432)]]]
IDS = [i if isinstance(i, str) else "-".join(map(str, i)) for i in INSTANCES]


def _states(field, count, seed):
    p = (BABYBEAR if field == 0 else KOALABEAR).p
    rng = np.random.default_rng(seed)
    x = rng.integers(0, p, size=(count, 16), dtype=np.uint64).astype(np.uint32)
    edge = np.array([0, 1, 2, p - 1, p - 2, p // 2, p // 2 + 1, 1 << 24, 1 << 27, (1 << 30) - 1],
                    np.uint32)
    h = (count + 1) // 2
    x[:h] = edge[rng.integers(0, edge.size, size=(h, 16))]
    x[0] = 0
    return x


@pytest.mark.parametrize("name", INSTANCES, ids=IDS)
@pytest.mark.parametrize("count", [1, 129, 1000])
def test_permutation_per_thread(orc, name, count):
    g, o = _instance(orc, name)
    x = _states(g.field.id, count, 3)
    got = to_host(g.permute(to_device(x).reshape(count, 16))).reshape(count, 16)
    want = np.stack([o.permute(s) for s in x])
    assert np.array_equal(got, want)


@pytest.mark.parametrize("name", INSTANCES, ids=IDS)
def test_transcript_chain(orc, name):
    g, o = _instance(orc, name)
    t, ot = DuplexTranscript.new(g), orc.Transcript(o)
    for m, n in [(8, 1), (40, 9), (3, 2), (13, 17)]:
        v = _states(g.field.id, 3, m)[1:].reshape(-1)[:m].copy() if m <= 32 else \
            _states(g.field.id, 4, m).reshape(-1)[:m].copy()
        t, got = t.observe_and_sample(to_device(v), n)
        ot.observe(v)
        assert np.array_equal(to_host(got), ot.sample(n))


@pytest.mark.parametrize("name", INSTANCES, ids=IDS)
@pytest.mark.parametrize("leaves", [2, 32, 256, 1024])
def test_tree_levels(orc, name, leaves):
    g, o = _instance(orc, name)
    x = _states(g.field.id, leaves, 5)
    _, layers = MerkleTree(g).commit(to_device(x[:, :8].copy()).reshape(leaves, 8))
    want = orc.merkle_commit(o, x[:, :8].copy().reshape(-1), leaves, 1, 8, 0)
    for lvl, w in enumerate(want):
        assert np.array_equal(to_host(layers[lvl]).reshape(-1), w.reshape(-1)), lvl

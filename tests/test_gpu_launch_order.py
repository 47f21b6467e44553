"""Kernels set up while the stream's previous kernel still runs: a chain of
launches over one reused buffer, with copies and fills between them, on two
streams joined by an event, and replayed from a captured graph, gives what the
same steps give with a synchronisation after each. Words are equal exactly."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from zorch_gb300 import _lib  # noqa: E402
from zorch_gb300.coding import ReedSolomon  # noqa: E402
from zorch_gb300.commit import MerkleTree, Poseidon2  # noqa: E402
from zorch_gb300.field import BABYBEAR, to_device  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    _lib.check(_lib.lib().zc_init(0), "init")


# message lengths: one launch a step, a few, and wide levels ended by narrow ones
SIZES = [4, 256, 1 << 13, 1 << 17]


def _chain(tree, code, x, step=lambda: None, reps=6):
    """Each repetition overwrites x with words of the last root, then encodes
    and commits it again."""
    roots = []
    for i in range(reps):
        cw = code.encode(x)
        step()
        root, _ = tree.commit(cw.reshape(-1, 2))
        step()
        roots.append(root.clone())
        x[:4].copy_(root[:4])
        x[-2:].fill_(i)
        step()
    return torch.stack(roots)


def _words(n):
    rng = np.random.default_rng(n)
    return to_device(rng.integers(0, BABYBEAR.p, size=n, dtype=np.uint64).astype(np.uint32))


@pytest.mark.parametrize("n", SIZES)
def test_chain_equals_synchronised_steps(n):
    tree, code = MerkleTree(Poseidon2.builtin(BABYBEAR)), ReedSolomon(n, 2, BABYBEAR)
    want = _chain(tree, code, _words(n), torch.cuda.synchronize)
    assert torch.equal(_chain(tree, code, _words(n)), want)

    side, x = torch.cuda.Stream(), _words(n)  # two streams, a hand-over between them
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        first = _chain(tree, code, x, reps=3)
    torch.cuda.current_stream().wait_stream(side)
    y = _words(n)
    y[:4].copy_(first[2][:4])
    y[-2:].fill_(2)
    assert torch.equal(x, y)
    assert torch.equal(first, want[:3])

    src, x = _words(n), torch.empty_like(_words(n))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x.copy_(src)
        got = _chain(tree, code, x)
    for _ in range(3):
        got.zero_()
        graph.replay()
        assert torch.equal(got, want)

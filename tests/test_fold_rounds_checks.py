"""What the fold rounds and the batched openings refuse before anything is
queued: shapes that do not fit one another, which the kernels would read past
the end of. The tensors live on the host, so nothing here can be launched."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

from zorch_gb300.coding import ReedSolomon  # noqa: E402
from zorch_gb300.commit import DigestLayers, Poseidon2, leaves_layout  # noqa: E402
from zorch_gb300.field import BABYBEAR  # noqa: E402
from zorch_gb300.pcs import CommittedLayer, open_layers, run_fold_rounds  # noqa: E402
from zorch_gb300.transcript import DuplexTranscript  # noqa: E402


def _z(*shape):
    return torch.zeros(shape, dtype=torch.int32)


def _cw(n):
    return n if torch.is_tensor(n) else _z(n)


def _layer(n, leaves, words=None):
    return CommittedLayer(_z(n), DigestLayers(_z(words or 2 * leaves - 1, 8), leaves))


@pytest.mark.parametrize("n,rounds,kw,match", [
    (12, 2, {}, "power of two"),
    (_z(16, 1), 2, {}, "codeword"),
    (_z(16, 2, 2), 2, {}, "codeword"),
    (16, 0, {}, "rounds"),
    (16, 5, {}, "rounds"),
    (16, 2, {"first_layer": _layer(16, 4)}, "first layer"),
    (16, 2, {"first_layer": _layer(16, 16)}, "first layer"),
    (16, 2, {"first_layer": _layer(16, 8, words=14)}, "first layer"),
    (16, 2, {"first_layer": _layer(32, 8)}, "first layer"),
    (16, 2, {"sumcheck": (_z(2, 4), _z(2, 4), _z(4), _z(2, 4))}, "sumcheck"),
    (16, 2, {"sumcheck": (_z(4, 4), _z(1, 4), _z(4), _z(2, 4))}, "sumcheck"),
    (16, 2, {"sumcheck": (_z(4, 4), _z(2, 4), _z(1), _z(2, 4))}, "sumcheck"),
    (16, 2, {"sumcheck": (_z(4, 4), _z(2, 4), _z(4), _z(1, 4))}, "sumcheck"),
])
@pytest.mark.parametrize("other", [False, True])
def test_shapes_that_do_not_fit(orc, n, rounds, kw, match, other):
    perm = Poseidon2.builtin()
    ei, et, ir, dg = orc.Poseidon2.babybear16().export_canonical()
    t = DuplexTranscript(Poseidon2.from_params(BABYBEAR, 7, et, ei, ir, dg) if other else perm,
                         torch.arange(34, dtype=torch.int32))
    code = ReedSolomon(8, 2, BABYBEAR)
    with pytest.raises(ValueError, match=match):
        run_fold_rounds(perm, code, _cw(n), rounds, 1, t, **kw)
    assert torch.equal(t.state, torch.arange(34, dtype=torch.int32))


@pytest.mark.parametrize("leaves,words,width", [(4, 7, 2), (16, 31, 2), (8, 14, 2), (8, 15, 3)])
def test_openings_that_do_not_fit(monkeypatch, leaves, words, width):
    from zorch_gb300 import commit

    monkeypatch.setattr(commit, "ptr", lambda t: t.data_ptr())
    cw = _z(16)
    spec = (leaves_layout(cw, 8, 2, 1, 8), DigestLayers(_z(words, 8), leaves), width, 0)
    with pytest.raises(ValueError, match="opening"):
        open_layers([spec], _z(3))

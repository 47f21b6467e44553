"""Batched tree commits over their work items: trees smaller than an item, of
exactly one, of one and a part of a wave, and families long enough that a CTA
claims several items, in one call, against one commit a tree. Words are equal
exactly."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from zorch_gb300 import _lib  # noqa: E402
from zorch_gb300.commit import Poseidon2, koalabear16_params  # noqa: E402
from zorch_gb300.field import BABYBEAR, KOALABEAR, ptr, stream_handle, to_device  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    _lib.check(_lib.lib().zc_init(0), "init")


# (log2 leaves, width, trees of the shape)
MIXES = [[(0, 1, 1)], [(0, 3, 5), (6, 9, 3), (7, 8, 2), (8, 1, 4)],
         [(9, 17, 700), (13, 2, 40), (3, 5, 1)], [(17, 1, 3), (12, 30, 2), (7, 2, 900)]]


@pytest.mark.parametrize("koala", [False, True])
@pytest.mark.parametrize("mix", range(len(MIXES)))
def test_batch_equals_single_commits(orc, mix, koala):
    field = KOALABEAR if koala else BABYBEAR
    perm = (koalabear16_params(orc.load_sp1_fixture()) if koala else Poseidon2.builtin(BABYBEAR))
    rng = np.random.default_rng(mix)
    L, st = _lib.lib(), stream_handle()
    jobs, data, got = (_lib.MerkleJob * len(MIXES[mix]))(), [], []
    for i, (log_l, w, count) in enumerate(MIXES[mix]):
        n = 1 << log_l
        x = rng.integers(0, field.p, size=(count, n * w), dtype=np.uint64).astype(np.uint32)
        data.append(to_device(x).reshape(count, n * w))
        got.append(torch.full((count, 2 * n, 8), -1, dtype=torch.int32, device="cuda"))
        jobs[i] = _lib.MerkleJob(_lib.Leaves(ptr(data[i]), n, 1, w, 0), ptr(got[i]), 0, count,
                                 n * w, 16 * n)
    ws = torch.empty(64, dtype=torch.int32, device="cuda")
    _lib.check(L.zc_merkle_commit_batch(perm.handle, jobs, len(jobs), ptr(ws), 256, st), "batch")
    for i, (log_l, w, count) in enumerate(MIXES[mix]):
        n = 1 << log_l
        want = torch.empty((2 * n - 1, 8), dtype=torch.int32, device="cuda")
        for t in sorted({0, count // 2, count - 1}):
            lv = _lib.Leaves(ptr(data[i][t]), n, 1, w, 0)
            _lib.check(L.zc_merkle_commit(perm.handle, lv, ptr(want), st), "single")
            assert torch.equal(got[i][t, :-1], want)
        assert bool((got[i][:, -1] == -1).all())  # the gap between trees is untouched

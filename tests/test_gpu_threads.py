"""Calls from several threads, each on its own stream, whose launches of one
kernel need different amounts of shared memory: every call runs and gives the
words it gives alone. (The limit that a launch may use is a property of the
kernel, set by whichever thread came last.)"""

from __future__ import annotations

import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from zorch_gb300 import _lib  # noqa: E402
from zorch_gb300.field import BABYBEAR, ptr, stream_handle, to_device  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    _lib.check(_lib.lib().zc_init(0), "init")


def _words(*shape, seed=1):
    x = np.random.default_rng(seed).integers(0, BABYBEAR.p, size=shape, dtype=np.uint64)
    return to_device(x.astype(np.uint32)).reshape(shape)


def _rlc(w):
    """A batching of w columns: 16 w bytes of shared memory."""
    cw, chal = _words(w, 4, seed=w), _words(12, 4, seed=w + 1)

    def call():
        out = torch.empty((4, 4), dtype=torch.int32, device="cuda")
        _lib.check(_lib.lib().zc_rlc_columns_ex(0, ptr(cw), 4, w, ptr(chal), 12, 0, 0, ptr(out),
                                                stream_handle()), "rlc")
        return out

    return call


def _encode(log_k):
    """An encode at blowup 2, buffers made once: as many calls a second as it takes."""
    x, L = _words(1 << log_k), _lib.lib()
    nb = L.zc_rs_encode_workspace_bytes(1, log_k, 1)
    bufs = {}

    def call():
        st = stream_handle()
        if st not in bufs:
            bufs[st] = [torch.empty(max(k, 1), dtype=torch.int32, device="cuda")
                        for k in (2 << log_k, nb // 4)]
        out, ws = bufs[st]
        _lib.check(L.zc_rs_encode(0, ptr(x), 1, log_k, 1, 0, 0, ptr(out), ptr(ws), nb, st),
                   "encode")
        return out

    return call


def _together(calls, count):
    """`count` runs of each call on a thread and stream of its own."""
    want = [c() for c in calls]
    torch.cuda.synchronize()
    errors = []

    def work(call, expect):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(count):
                    got = call()
                ok = torch.equal(got, expect)
            if not ok:
                errors.append("other words than alone")
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(c, w)) for c, w in zip(calls, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors


def test_batching_of_different_widths():
    _together([_rlc(4096), _rlc(3200), _rlc(4096), _rlc(3600)], 4000)


@pytest.mark.parametrize("logs", [(13, 4), (13, 12), (15, 14), (20, 15), (24, 14)])
def test_encodes_of_different_lengths(logs):
    _together([_encode(k) for k in logs * 2], 200 if logs[0] > 16 else 6000)

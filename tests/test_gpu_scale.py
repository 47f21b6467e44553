"""zc_scale: every word times one Montgomery scalar, at one word, around a block and
past one sweep of the grid (152 x 16 blocks of 256), in place too."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from zorch_gb300 import _lib  # noqa: E402
from zorch_gb300.field import BABYBEAR, KOALABEAR, ptr, stream_handle, to_device, to_host  # noqa: E402


@pytest.mark.parametrize("n", [1, 3, 255, 257, 152 * 16 * 256 + 1])
@pytest.mark.parametrize("field", [BABYBEAR, KOALABEAR], ids=lambda f: f.name)
def test_scale(field, n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p, rinv = field.p, pow(1 << 32, field.p - 2, field.p)
    x = np.random.default_rng(n).integers(0, p, size=n, dtype=np.uint64)
    x[:4] = [0, 1, p - 1, p // 2][:n]
    d = to_device(x.astype(np.uint32))
    for s in (0, 1, field.mont(1), p - 1, field.inv_mont(field.mont(1 << 20))):
        out = torch.empty_like(d)
        L = _lib.lib()
        _lib.check(L.zc_scale(field.id, ptr(d), ptr(out), n, s, stream_handle()), "scale")
        want = x * np.uint64(s * rinv % p) % np.uint64(p)  # both below 2^31
        assert np.array_equal(to_host(out), want.astype(np.uint32))
        same = d.clone()
        _lib.check(L.zc_scale(field.id, ptr(same), ptr(same), n, s, stream_handle()), "scale")
        assert torch.equal(same, out)

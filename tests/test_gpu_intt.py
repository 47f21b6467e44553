"""The inverse transform in one pass pair (zc_intt) against its definition over
the forward one, (1/k) NTT(x)[-i mod k], on every path of the transform: a
single shared-memory pass, the four-step passes and their wide build, one
column and many, both fields, and extend() (inverse, then the coset code)
against encode() of the recovered coefficients. Words are equal exactly."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from zorch_gb300 import _lib  # noqa: E402
from zorch_gb300.coding import ReedSolomon, intt, ntt  # noqa: E402
from zorch_gb300.field import BABYBEAR, KOALABEAR, to_device, to_host  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    _lib.check(_lib.lib().zc_init(0), "init")


def _words(field, *shape):
    rng = np.random.default_rng(shape[-1])
    x = rng.integers(0, field.p, size=shape, dtype=np.uint64).astype(np.uint32)
    x[..., :2] = field.p - 1
    return to_device(x).reshape(shape)


# (columns, log_k): single pass to 2^12, four-step, and two tiles per SM or more
SIZES = [(1, 0), (3, 1), (2, 5), (5, 11), (1, 12), (1, 13), (3, 14), (7, 16), (1, 17), (40, 17),
         (80, 16), (2, 20), (320, 14)]


@pytest.mark.parametrize("field", [BABYBEAR, KOALABEAR], ids=lambda f: f.name)
@pytest.mark.parametrize("w,log_k", SIZES)
def test_intt_is_its_definition(field, w, log_k):
    k = 1 << log_k
    x = _words(field, w, k)
    got = intt(field, x)
    y = to_host(ntt(field, x)).reshape(w, k).astype(np.uint64)
    kinv = np.uint64(pow(k, field.p - 2, field.p))
    want = y[:, (-np.arange(k)) % k] * kinv % np.uint64(field.p)
    assert np.array_equal(to_host(got).reshape(w, k), want.astype(np.uint32))
    assert torch.equal(ntt(field, got), x)


@pytest.mark.parametrize("field", [BABYBEAR, KOALABEAR], ids=lambda f: f.name)
@pytest.mark.parametrize("w,log_k,log_b", [(1, 3, 1), (3, 11, 2), (5, 14, 1), (33, 16, 1)])
def test_extend(field, w, log_k, log_b):
    code = ReedSolomon(1 << log_k, 1 << log_b, field, coset_shift=field.generator)
    coeffs = _words(field, w, 1 << log_k)
    assert torch.equal(code.extend(ntt(field, coeffs)), code.encode(coeffs))

"""The multilinear kernels against the oracle at the sizes where their splits
change: eq tables around six and twelve variables, evaluations with column
counts around the four a CTA takes, batchings with odd column counts, offsets
and accumulation, and the limb transposes. Words at the ends of [0, p) are
among the inputs; equality is exact."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from zorch_gb300 import _lib  # noqa: E402
from zorch_gb300.field import BABYBEAR, KOALABEAR, ptr, stream_handle, to_device, to_host  # noqa: E402

FIELDS = [BABYBEAR, KOALABEAR]


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    _lib.check(_lib.lib().zc_init(0), "init")


def _words(field, *shape, seed=1):
    rng = np.random.default_rng(seed)
    x = rng.integers(0, field.p, size=shape, dtype=np.uint64).astype(np.uint32)
    edge = np.array([0, 1, field.p - 1, field.p // 2, field.p // 2 + 1], np.uint32)
    m = rng.random(shape) < 0.3
    x[m] = edge[rng.integers(0, edge.size, size=int(m.sum()))]
    return x


def _dev(x):
    return to_device(x).reshape(x.shape)


def _ws(nb):
    return torch.empty(max((nb + 15) // 4, 4), dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("field", FIELDS, ids=lambda f: f.name)
@pytest.mark.parametrize("m", [0, 1, 2, 5, 6, 7, 11, 12, 13, 14])
def test_eq_tables(orc, field, m):
    L = _lib.lib()
    z = _words(field, max(m, 1), 4, seed=m)[:m]
    out = torch.empty((1 << m, 4), dtype=torch.int32, device="cuda")
    nb = L.zc_eq_expand_workspace_bytes(m)
    ws, zd = _ws(nb), _dev(z) if m else None
    _lib.check(L.zc_eq_expand(field.id, ptr(zd), m, ptr(out), ptr(ws), nb,
                              stream_handle()))
    want = orc.eq_expand(field.id, z) if m else np.array([[field.one_mont, 0, 0, 0]], np.uint32)
    assert np.array_equal(to_host(out), want)


@pytest.mark.parametrize("field", FIELDS, ids=lambda f: f.name)
@pytest.mark.parametrize("w,m", [(1, 1), (2, 5), (3, 8), (4, 9), (5, 12), (8, 13), (9, 14), (1, 16)])
def test_eval_columns(orc, field, w, m):
    L = _lib.lib()
    cols, z = _words(field, w, 1 << m, seed=w), _words(field, m, 4, seed=m)
    out = torch.empty((w, 4), dtype=torch.int32, device="cuda")
    nb = L.zc_eval_mle_workspace_bytes(w, m)
    ws, cd, zd = _ws(nb), _dev(cols), _dev(z)
    _lib.check(L.zc_eval_mle(field.id, ptr(cd), w, m, ptr(zd), ptr(out), ptr(ws), nb,
                             stream_handle()))
    assert np.array_equal(to_host(out), orc.eval_mle_base(field.id, cols, z))


@pytest.mark.parametrize("field", FIELDS, ids=lambda f: f.name)
@pytest.mark.parametrize("w,off,n", [(1, 0, 1), (2, 0, 300), (3, 1, 257), (5, 2, 1000), (8, 0, 4096),
                                     (7, 9, 33), (130, 3, 64)])
def test_batching(orc, field, w, off, n):
    L = _lib.lib()
    nbv = (w + off - 1).bit_length()
    cw, vals = _words(field, w, n, seed=w), _words(field, w, 4, seed=2)
    chal = _words(field, max(nbv, 1), 4, seed=3)
    chd, cwd, vd = _dev(chal), _dev(cw), _dev(vals)
    wt = orc.eq_expand(field.id, chal[:nbv]) if nbv else np.array([[field.one_mont, 0, 0, 0]],
                                                                  np.uint32)
    start = _words(field, n, 4, seed=4)
    for acc in (0, 1):
        out, claim = _dev(start), _dev(start[0])
        _lib.check(L.zc_rlc_columns_ex(field.id, ptr(cwd), n, w, ptr(chd), nbv, off, acc,
                                       ptr(out), stream_handle()))
        _lib.check(L.zc_rlc_values(field.id, ptr(vd), w, ptr(chd), nbv, off, acc,
                                   ptr(claim), stream_handle()))
        want = start.copy() if acc else np.zeros((n, 4), np.uint32)
        orc.LIB.orc_rlc_columns_ex(field.id, cw.reshape(-1), n, w, chal.reshape(-1), nbv, off, acc,
                                   want.reshape(-1))
        assert np.array_equal(to_host(out), want)
        c = start[0] if acc else np.zeros(4, np.uint32)
        for i in range(w):
            c = orc.ef4_add(field.id, c, orc.ef4_mul(field.id, wt[off + i], vals[i]))
        assert np.array_equal(to_host(claim), c)


@pytest.mark.parametrize("n", [1, 2, 255, 4096, 70001])
def test_limb_transposes(n):
    L, x = _lib.lib(), _dev(_words(KOALABEAR, n, 4))
    limbs, back = torch.empty((4, n), dtype=torch.int32, device="cuda"), torch.empty_like(x)
    _lib.check(L.zc_ef4_limbs(ptr(x), n, 1, ptr(limbs), stream_handle()))
    assert torch.equal(limbs, x.t())
    _lib.check(L.zc_ef4_limbs(ptr(limbs), n, 0, ptr(back), stream_handle()))
    assert torch.equal(back, x)
